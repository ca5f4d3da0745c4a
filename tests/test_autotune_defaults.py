"""BatchSolver.autotune with its defaults leaves the multigrid's coarse tile at the library's default: the
tile it sets back is the one a batch had before it was tuned."""
import pathlib
import re

from vebisph_gb300.solver import BatchSolver

CSRC = pathlib.Path(__file__).resolve().parent.parent / "vebisph_gb300" / "csrc"


class _Instance:
    def __init__(self, coarse):
        self.rows, self.coarse = 1, coarse

    def set_solver_grid(self, rows):
        self.rows = rows

    def set_coarse_block_rows(self, rows):
        self.coarse = rows


def test_defaults_keep_the_coarse_tile():
    default = int(re.search(r"MG_BLOCK_ROWS = (\d+);", (CSRC / "vebi_common.cuh").read_text()).group(1))
    b = object.__new__(BatchSolver)  # no library, no GPU: the steps' times are given
    b.instances = [_Instance(default) for _ in range(3)]
    tried = []

    def step(n):
        i = b.instances[0]
        tried.append((i.rows, i.coarse))
        return {1: 4.0, 2: 3.0, 4: 1.0, 8: 2.0}[i.rows], []

    b.step = step
    got = b.autotune()
    assert got["rows_per_thread"] == 4 and {i.rows for i in b.instances} == {4}
    assert got["coarse_block_rows"] == default and {i.coarse for i in b.instances} == {default}
    assert {c for _, c in tried} == {default}
