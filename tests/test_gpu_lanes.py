"""Pair sums by eight lanes a row (small domains) and by a thread a row, at the edges of both: part
of a block, sizes either side of the lines at 10,000 and 30,000 rows."""
import numpy as np
import pytest

from tests.parity import EXACT_ELL, compare_step, partner
from vebisph_gb300 import abi, cases

pytestmark = pytest.mark.gpu

SUMS = ("gradu_x", "gradu_y", "gradv_x", "gradv_y", "gradth_x", "gradth_y", "ustar_x", "ustar_y", "theta_star")


def _case(name, const_mod=2):
    kind, n = name.split(":")
    c = (cases.cavity if kind == "cavity" else cases.poiseuille)(int(n), seed=int(n))
    rng = np.random.default_rng(int(n))
    half = len(c.u) // 2  # fluid; the walls, which follow it, stay at rest
    c.u[:half] = 0.01 * rng.standard_normal((half, 2))
    c.const_mod = const_mod
    c.itermax = 2  # the pair sums need no solve
    return c


@pytest.mark.parametrize("const_mod", [1, 2])
@pytest.mark.parametrize("name", ["channel:4", "channel:5", "channel:98", "channel:99", "cavity:171", "cavity:172"])
def test_fp64_sums_equal_the_oracle(built, name, const_mod):
    from oracle.oracle import OracleSolver
    from vebisph_gb300.solver import StepSolver
    case = _case(name, const_mod)
    gpu, ref = StepSolver(case), OracleSolver(case)
    gpu.step(), ref.step()
    rep = compare_step(gpu, ref, case)
    for nm in (*EXACT_ELL, *SUMS, "ppe_B"):
        assert rep[nm][0] <= rep[nm][1], (nm, rep[nm])
    gpu.close()
    ref.close()


@pytest.mark.parametrize("name", ["channel:4", "channel:98", "channel:99", "cavity:171", "cavity:172"])
def test_fp32_sums_close_to_fp64(built, name):
    """FP32 sums of some 44 terms, of which a few digits cancel: 44 * 2**-24 * 10 of the field's size."""
    from vebisph_gb300.solver import StepSolver
    a, b = StepSolver(_case(name), precision=abi.PREC_MIXED), StepSolver(_case(name), precision=abi.PREC_FP64)
    a.step(), b.step()
    for nm in (*SUMS, "ppe_B"):
        x, y = a.get(nm), b.get(nm)
        scale = max(np.abs(y).max(), np.abs(b.get(partner(nm))).max() if partner(nm) else 0.0)
        assert scale > 0 or np.array_equal(x, y), nm
        assert np.abs(x - y).max() <= 44 * 2.0**-24 * 10 * scale, (nm, np.abs(x - y).max() / scale)
    a.close()
    b.close()


@pytest.mark.parametrize("name", ["dam:4", "dam:33", "dam:118", "dam:119", "surface:75"])
def test_free_surface_sums_equal_the_oracle(built, name):
    from oracle.oracle import OracleSolver
    from vebisph_gb300.solver import StepSolver
    kind, n = name.split(":")
    case = (cases.dam_break if kind == "dam" else cases.free_surface_periodic)(int(n), seed=int(n))
    case.itermax = 2
    gpu, ref = StepSolver(case), OracleSolver(case)
    gpu.step(), ref.step()
    assert np.array_equal(gpu.get("n_surf")[: case.npfb], ref.get("n_surf")[: case.npfb])
    for nm in ("conc", "div_r"):
        a, b = gpu.get(nm), ref.get(nm)
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max(), nm
    rep = compare_step(gpu, ref, case)
    for nm in ("ushift_x", "ushift_y", *SUMS):
        assert rep[nm][0] <= rep[nm][1], (nm, rep[nm])
    gpu.close()
    ref.close()
