"""The PPE solvers whose rows are spread over all SMs (vebi_resident.cu, vebi_noalloc.cu), their kernels
compiled for the CPU from the same sources (tests/emulated): a solve gives the same bits whether the
blocks keep within one block barrier of one another or one of them, each in its turn, runs ahead to
the next grid barrier while the others have not yet read what the last one was for."""
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    out = tmp_path_factory.mktemp("emulated") / "solvers"
    subprocess.run(["g++", "-x", "c++", "-O1", "-std=c++17", "-ffp-contract=off", "-pthread", "-Wno-attributes",
                    "-fno-extern-tls-init",  # the dynamic shared memory has no initialiser
                    "-I", str(ROOT / "tests" / "emulated"), "-I", str(ROOT / "vebisph_gb300" / "csrc"),
                    "-I", str(ROOT / "include"), "-o", str(out), str(ROOT / "tests" / "emulated" / "solvers.cpp")],
                   check=True)
    return out


def _run(exe, *args):
    r = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr


# one group of 32 rows an SM (the products take off the mean themselves), a few, and blocks of more than 128
# rows, whose slots come from memory
@pytest.mark.parametrize("rows,sms", [(200, 8), (250, 4), (600, 3)])
@pytest.mark.parametrize("closed,warm", [(1, 0), (1, 1), (0, 0), (0, 1)])
def test_resident_solve_whichever_block_is_ahead(exe, rows, sms, closed, warm):
    _run(exe, "resident", rows, sms, closed, warm)


# more rows than one SM's 512, so that one SM takes the persistent kernel: two groups an SM, the last SM's
# partly empty, and five
@pytest.mark.parametrize("rows,sms", [(513, 12), (700, 5)])
@pytest.mark.parametrize("closed", [1, 0])
def test_noalloc_solve_whichever_block_is_ahead(exe, rows, sms, closed):
    _run(exe, "noalloc", rows, sms, closed)
