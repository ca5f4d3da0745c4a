"""The mirrors of a step (selected for all patches and circles at once, vebi_geom.cu) against the
oracle's, which makes them patch by patch: the same mirrors in the same order, bit for bit."""
import numpy as np
import pytest

from vebisph_gb300 import cases

pytestmark = pytest.mark.gpu


def _two_circles(c):
    # a second circle a little smaller than the first: the particles near both have two images
    c.c_centre = np.vstack([c.c_centre, c.c_centre])
    c.c_radius = np.array([c.c_radius[0], c.c_radius[0] - 2.0 * c.dx])
    c.c_omega = np.array([0.3, -0.2])
    c.c_vel = np.array([[0.1, 0.0], [0.0, 0.2]])
    c.c_thermal = np.array([0.5, 0.25])
    return c


CASES = {
    # less than a word of particles, one past it; one block, one past it; the larger blocks, at a
    # remainder (448^2 particles are 196 of them)
    "channel5": lambda: cases.poiseuille(5, seed=1),
    "channel6": lambda: cases.poiseuille(6, seed=2),
    "channel16": lambda: cases.poiseuille(16, seed=3),
    "cavity17": lambda: cases.cavity(17, seed=4),
    "channel448": lambda: cases.poiseuille(448, seed=5),
    "dam_break33": lambda: cases.dam_break(33, seed=6),
    "cylinder": lambda: cases.cylinder(8.0e3, seed=7),
    "two_circles": lambda: _two_circles(cases.cylinder(8.0e3, seed=8)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_mirrors_equal_the_oracle(built, name):
    from oracle.oracle import OracleSolver
    from vebisph_gb300.solver import StepSolver
    case = CASES[name]()
    case.itermax = 2  # the mirrors precede the solve
    gpu, ref = StepSolver(case), OracleSolver(case)
    sg, so = gpu.step(), ref.step()
    assert sg["nmirror"] == so["nmirror"] > 0
    for nm in ("irelation", "vrelation", "rsx", "rsy", "dP_mp"):
        a, b = gpu.get(nm), ref.get(nm)
        assert a.shape == b.shape and np.array_equal(a, b), nm
    gpu.close()
    ref.close()


@pytest.mark.parametrize("name", ["channel5", "channel16", "cavity17", "dam_break33", "two_circles"])
def test_matrix_of_rows_with_mirrors(built, name):
    """k_ppe_mirror_rows: a mirror's term goes to its parent's column, out of the diagonal for the
    row's own mirror, and into the right-hand side.  A row near a free surface is scaled by a factor
    with a cosine, which differs from the oracle's in the last place."""
    from oracle.oracle import OracleSolver
    from tests.parity import EXACT_ELL, compare_step
    from vebisph_gb300.solver import StepSolver
    case = CASES[name]()
    case.itermax = 2
    gpu, ref = StepSolver(case), OracleSolver(case)
    gpu.step(), ref.step()
    rep = compare_step(gpu, ref, case)
    for nm in (*EXACT_ELL, "ppe_diag", "ppe_B"):
        tol = 2.0**-50 if case.i_open_domain == 1 and nm == "ppe_val" else rep[nm][1]
        assert rep[nm][0] <= tol, (nm, rep[nm])
    gpu.close()
    ref.close()


@pytest.mark.parametrize("const_mod", [1, 2])
@pytest.mark.parametrize("name", ["cylinder", "two_circles"])
def test_force_on_circles(built, name, const_mod):
    """k_circle_terms, Newtonian and viscoelastic: within the pressure's tolerance of the oracle."""
    from oracle.oracle import OracleSolver
    from vebisph_gb300.solver import StepSolver
    case = CASES[name]()
    case.const_mod = const_mod
    gpu, ref = StepSolver(case), OracleSolver(case)
    fg, fo = np.array(gpu.step()["circle_force"]), np.array(ref.step()["circle_force"])
    assert np.abs(fo).max() > 0 and np.abs(fg - fo).max() <= 1e-5 * np.abs(fo).max(), (fg, fo)
    gpu.close()
    ref.close()
