"""The FP64 PPE solve with its rows spread over all SMs (vebi_resident.cu) against the persistent
kernel it stands in for: both sum in the same order, so a step agrees bit for bit.  A batch's
instances keep the persistent kernel, so a batch of one is the reference."""
import numpy as np
import pytest

from vebisph_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _warm(c):
    c.ppe_warm_start = 1
    return c


def _capped(c):
    c.itermax = 7
    return c


CASES = {
    # row counts at the edges: one group of 32 rows or a few, 32 virtual blocks and one more, blocks of more
    # than 128 rows (slots from L2), the largest system that fits and one that does not
    "channel6": lambda: cases.poiseuille(6, seed=1),
    "channel40": lambda: cases.poiseuille(40, seed=2),
    "channel89": lambda: cases.poiseuille(89, seed=3),
    "channel92": lambda: cases.poiseuille(92, seed=4),
    "cylinder21k": lambda: cases.cylinder(2.1e4, Wi=0.6, seed=5),
    "channel195": lambda: cases.poiseuille(195, seed=6),
    "channel199": lambda: cases.poiseuille(199, seed=7),
    "free_surface_open": lambda: cases.free_surface_periodic(75, seed=8),
    "dam_break_open": lambda: cases.dam_break(33, seed=9),
    "warm": lambda: _warm(cases.poiseuille(45, seed=10)),
    "warm_open": lambda: _warm(cases.dam_break(24, seed=11)),
    "capped": lambda: _capped(cases.cavity(50, seed=12)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_resident_solve_equals_the_persistent_one(built, name):
    from vebisph_gb300.solver import BatchSolver, StepSolver
    one = StepSolver(CASES[name](), precision=abi.PREC_FP64)
    ref = BatchSolver([CASES[name]()], precision=abi.PREC_FP64)
    for step in range(2):
        s = one.step()
        _, st = ref.step(1)
        assert (s["LS_iters"], s["LS_residual"], s["warnings"]) == \
            (st[0]["LS_iters"], st[0]["LS_residual"], st[0]["warnings"]), step
        for nm in ("p", "ux", "uy", "rx", "ry"):
            a, b = one.get(nm), ref.instances[0].get(nm)
            assert np.array_equal(a, b), (step, nm)
    one.close()
    ref.close()
