"""Products, quotients and square roots on the integer and FP32 pipes (vebi_fp64.cuh is host/device)
against the processor's, bit for bit, over 4 million seeded operands of every class; and, on the
GPU, the pairs that only one of their particles lists."""
import pathlib
import shutil
import subprocess

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent


def test_results_are_the_processors(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = tmp_path / "check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "vebisph_gb300" / "csrc"),
                    "-o", str(exe), str(ROOT / "tests" / "fp64" / "check.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def _past_the_right_side(m=24, seed=3):
    """A water column across an open right side (patch type 0), out to the last cell column, whose
    particles the reference gives no western cells."""
    from vebisph_gb300 import cases
    c = cases.dam_break(m, seed=seed)
    c.b_type = np.array([1, 0, 1, 1])
    c.r[c.nbS:, 0] += 1.0 + 1.40 * 3.0 * c.h - c.r[c.nbS:, 0].max()
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [8, 4, 1])
def test_weights_of_one_sided_pairs(built, lanes):
    """ij_link, the weights and the correction matrix are the oracle's bit for bit, whichever number of
    lanes a row gets."""
    from oracle.oracle import OracleSolver
    from vebisph_gb300.solver import StepSolver
    # particles of the free-surface column, repeated downwards only in number: the rule is on npfb
    c = _past_the_right_side({8: 24, 4: 150, 1: 290}[lanes])
    assert {8: c.npfb <= 40000, 4: 40000 < c.npfb <= 150000, 1: c.npfb > 150000}[lanes]
    c.itermax = 3
    gpu, ref = StepSolver(c), OracleSolver(c)
    gpu.step(), ref.step()
    cnt = ref.get("ij_count")
    assert np.array_equal(gpu.get("ij_count"), cnt)
    k = int(cnt.max())
    mask = np.arange(k)[:, None] < cnt[None, :]
    link = ref.get("ij_link").reshape(-1, c.npfb)[:k]
    i, kk = np.nonzero((mask & (link < c.npfb)).T)
    pairs = set(zip(i.tolist(), link.T[i, kk].tolist())) if lanes == 8 else None
    if pairs is not None:  # the case does hold pairs that only one particle lists
        assert any((j, i) not in pairs for i, j in pairs)
    for nm in ("ij_link", "w_Gx", "w_Gy", "w_L"):
        a, b = gpu.get(nm).reshape(-1, c.npfb)[:k], ref.get(nm).reshape(-1, c.npfb)[:k]
        assert np.array_equal(a[mask], b[mask]), nm
    for nm in ("kgcm11", "kgcm21", "kgcm12", "kgcm22"):
        assert np.array_equal(gpu.get(nm), ref.get(nm)), nm
    for nm in ("gradC_x", "gradC_y", "ushift_x", "ushift_y"):
        a, b = gpu.get(nm), ref.get(nm)
        assert np.abs(a - b).max() <= 1e-13 * np.abs(b).max(), nm
    gpu.close()
    ref.close()
