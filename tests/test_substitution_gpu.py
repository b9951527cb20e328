"""FAST triangular solves with infinities and NaN among the right-hand sides, against the
reference's sequence in numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(t, b, trans):
    """Substitution in the reference's order (divide, subtract from all later rows)."""
    n = len(t)
    m = t.T if trans else t
    x = b.copy()
    with np.errstate(all="ignore"):
        for i in (range(n) if not trans else range(n - 1, -1, -1)):
            x[i] = x[i] / m[i, i]
            later = slice(i + 1, n) if not trans else slice(0, i)
            x[later] -= m[later, i][:, None] * x[i][None, :]
    return x


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 70])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("trans", [0, 1])
def test_fast_substitution_non_finite(gpu_lla, dtype, n, dense, trans):
    """Signed infinities stay what the division gives, whatever the diagonal (a power of two, whose
    reciprocal is exact, or not), NaN spreads no further than in the reference, and a row whose
    quotient alone would overflow takes its coupling first."""
    import torch
    rng = np.random.default_rng(n)
    t = np.diag(rng.choice([1.0, -2.0, 0.25, 3.0, -0.7, 1.3], n)) + (np.tril(rng.uniform(0.1, 0.2, (n, n)), -1) if dense else 0)
    b = rng.uniform(1, 2, (n, 6))
    b[n // 2, 0] = np.inf
    b[n // 3, 1] = -np.inf
    b[n - 1, 2] = np.nan
    b[0, 3], b[n - 1, 3] = np.inf, -np.inf
    if n > 1 and dense:  # column 4: big in the first row, then big - 1 * big = 0 over a tiny diagonal in the last
        big, tiny = (1e300, 1e-20) if dtype == np.float64 else (1e30, 1e-12)
        i, j = (0, n - 1) if not trans else (n - 1, 0)
        t[1:n - 1, 0] = t[n - 1, 1:n - 1] = 0
        t[i, i], t[j, j], t[n - 1, 0] = 1.0, tiny, 1.0
        b[:, 4] = 0
        b[[0, n - 1], 4] = big
    t, b = t.astype(dtype), b.astype(dtype)
    want = _solve(t, b, trans)
    L = torch.from_numpy(np.ascontiguousarray(t.T)).cuda().T
    X = torch.zeros(b.shape[1], n + 3, dtype=L.dtype, device="cuda").T[:n]
    X.copy_(torch.from_numpy(b))
    gpu_lla.trsm_device(L, X, trans, algo=gpu_lla.ALGO_FAST)
    gpu_lla.device_status()
    got = X.cpu().numpy()
    for c in range(b.shape[1]):
        assert (np.isnan(got[:, c]) == np.isnan(want[:, c])).all(), c
        inf = np.isinf(want[:, c])
        assert (np.isinf(got[:, c]) == inf).all() and (got[inf, c] == want[inf, c]).all(), c
    # a finite column: n products and a scaled row each, in any order
    assert np.isfinite(want[:, 5]).all()
    base = (t.T if trans else t).astype(np.float64)
    r = np.abs(base @ got[:, 5].astype(np.float64) - b[:, 5])
    den = np.abs(base) @ np.abs(got[:, 5].astype(np.float64)) + np.abs(b[:, 5])
    assert (r <= 4 * max(n, 4) * np.finfo(dtype).eps * den).all()
