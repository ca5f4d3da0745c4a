"""The solvers' grid barrier gives up after the 2 to 4 seconds that are promised: SPIN_LIMIT times the
time of a poll, measured on the same barrier with a short limit (0.2 s) that runs out."""
import ctypes as C
import pathlib
import re

import pytest

from vebisph_gb300 import abi

pytestmark = pytest.mark.gpu

CSRC = pathlib.Path(__file__).resolve().parent.parent / "vebisph_gb300" / "csrc"


@pytest.mark.parametrize("blocks", [2, 64])
def test_bound_of_the_grid_barrier(built, blocks):
    lib = abi.load_library()
    limit = 1 << int(re.search(r"SPIN_LIMIT = 1ull << (\d+);", (CSRC / "vebi_solver.cuh").read_text()).group(1))
    st, ms = C.c_int32(-1), C.c_double(0.0)
    assert lib.vebi_test_barrier_timeout(blocks, 1 << 20, C.byref(st), C.byref(ms)) == 0, lib.vebi_last_error()
    assert st.value == abi.STATUS["VEBI_ERR_TIMEOUT"]
    seconds = ms.value * 1.0e-3 * limit / (1 << 20)
    assert 1.5 < seconds < 4.5, seconds
