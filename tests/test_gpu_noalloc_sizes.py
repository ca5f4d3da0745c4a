"""vebi_ppe_solve_noalloc at the edges of its rows' split: a few rows, a group of 32 and one more,
a virtual block of 256 and one more, every number of groups per SM up to the largest system, and
rows with more slots than a block's shared memory holds.

The systems are graph Laplacians (a ring and random chords, symmetric weights), which BiCGSTAB
solves in a few dozen iterations; the stopping rule bounds the recursive residual by 1e-8 of the
first one, and the true residual is allowed 100 times that."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _laplacian(n, chords, seed):
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    a = np.concatenate([i] + [i] * chords)
    b = np.concatenate([(i + 1) % n] + [(i + 1 + rng.integers(1, max(n - 2, 2), n)) % n for _ in range(chords)])
    w = -rng.uniform(0.5, 1.5, a.size)
    keep = a != b
    a, b, w = a[keep], b[keep], w[keep]
    row, col, val = np.concatenate([a, b]), np.concatenate([b, a]), np.concatenate([w, w])
    o = np.argsort(row, kind="stable")
    row, col, val = row[o], col[o], val[o]
    cnt = np.bincount(row, minlength=n)
    slot = np.arange(row.size) - np.repeat(np.cumsum(cnt) - cnt, cnt)
    ecol, eval_ = np.zeros((cnt.max(), n), np.int32), np.zeros((cnt.max(), n))
    ecol[slot, row], eval_[slot, row] = col, val
    return cnt.astype(np.int32), ecol, eval_, -eval_.sum(0), rng


@pytest.mark.parametrize("closed", [1, 0])
@pytest.mark.parametrize("n,chords", [(3, 0), (32, 3), (33, 3), (256, 4), (257, 4), (4865, 20), (9729, 20),
                                      (38913, 20), (65536, 30)])
def test_residual(built, n, chords, closed):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device visible to torch")
    from vebisph_gb300 import abi
    lib = abi.load_library()
    cnt, col, val, diag, rng = _laplacian(n, chords, n + closed)
    rhs = 100.0 * rng.standard_normal(n)
    fixed = np.zeros(n, bool)
    if closed:
        rhs -= rhs.mean()
    else:
        fixed[:: max(n // 3, 1)] = True
        diag[fixed] = 1.0e30
    g = [torch.from_numpy(np.ascontiguousarray(q)).cuda() for q in (cnt, col, val, diag, rhs)]
    x = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    iters, resid = C.c_int32(0), C.c_double(0.0)
    st = lib.vebi_ppe_solve_noalloc(*[q.data_ptr() for q in g], x.data_ptr(), n, n, closed, 1.0e-8, 1000,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream), C.byref(iters),
                                    C.byref(resid))
    assert st == 0, lib.vebi_last_error()
    assert 1 <= iters.value < 1000
    p = x.cpu().numpy()
    r = rhs - diag * p - (val * p[col]).sum(0)
    free = ~fixed
    assert np.linalg.norm(r[free]) <= 1.0e-6 * np.linalg.norm(rhs), (iters.value, resid.value)
    assert np.abs(p[fixed]).max(initial=0.0) <= 1.0e-20
