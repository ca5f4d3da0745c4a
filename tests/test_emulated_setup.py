"""Set-up kernels of the step, compiled for the CPU from their sources (tests/emulated), at what no run of
the library on a GPU singles out: the multigrid levels by a warp and by a thread per coarse row, the
coarsest level's inverse with exchanged rows, and corners whose lists of mirrors and particles overflow."""
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent


def _build(out, *defines):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    subprocess.run(["g++", "-x", "c++", "-O1", "-std=c++17", "-ffp-contract=off", "-pthread", "-Wno-attributes",
                    *defines, "-I", str(ROOT / "tests" / "emulated"), "-I", str(ROOT / "vebisph_gb300" / "csrc"),
                    "-I", str(ROOT / "include"), "-o", str(out), str(ROOT / "tests" / "emulated" / "setup.cpp")],
                   check=True)
    return out


@pytest.fixture(scope="module")
def multigrid(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("emulated") / "multigrid")


@pytest.fixture(scope="module")
def corners(tmp_path_factory):
    """The library's list length, one that overflows at once and one that the first corner's mirrors overflow."""
    d = tmp_path_factory.mktemp("emulated")
    return [_build(d / f"corners{n}", f"-DCORNER_LIST={n}") for n in (4096, 3, 110)]


def _run(exe, *args):
    r = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr
    return r.stdout


@pytest.mark.parametrize("gx,gy", [(13, 9), (6, 5), (3, 2), (1, 1)])
def test_levels_by_a_warp_and_by_a_thread(multigrid, gx, gy):
    """Every level's columns, values and diagonal are the same bits, and rows too full for a level are
    reported by both."""
    _run(multigrid, "levels", gx, gy, 7)


@pytest.mark.parametrize("n", [1, 2, 5, 31, 32])
def test_coarse_inverse(multigrid, n):
    _run(multigrid, "inverse", n, 11)


@pytest.mark.parametrize("types", ["1212", "2121", "1111", "2222"])
def test_corners_with_overflowing_lists(corners, types):
    want, *others = [_run(exe, "mirrors", types, 3) for exe in corners]
    assert int(want.split()[0]) > 400
    assert all(o == want for o in others)
