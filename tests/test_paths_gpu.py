"""Device paths at the sizes where they can go wrong (edges of tiles,
remainders, both sides of a dispatch rule), against FP64 references."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    return torch


def _spd(torch, n, shift, seed):
    """G G^T / n + shift I (kappa about 4 / shift), FP64, symmetric."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    G = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    A = G @ G.T / n
    A = (A + A.T) * 0.5
    A.diagonal().add_(shift)
    return A, g


@pytest.mark.parametrize("n,m", [(65, 1), (600, 3), (1000, 64), (1500, 70)])
@pytest.mark.parametrize("shift", [1.0, 0.01])
def test_refined_slices_of_well_conditioned_systems_converge(gpu_lla, n, m, shift):
    """One correction takes a well-conditioned system to its target: the exact-slice
    residual has to resolve that error (no stall, no fallback to plain FP64)."""
    torch = _torch()
    A, g = _spd(torch, n, shift, n + m)
    B = torch.randn(m, n, dtype=torch.float64, device="cuda", generator=g).T
    X = torch.empty(m, n, dtype=torch.float64, device="cuda").T
    rep = gpu_lla.posv_refined_device(A.T, B, X, residual="slices")
    torch.cuda.synchronize()
    assert rep["converged"] == 1 and rep["fell_back"] == 0 and rep["iterations"] <= 3, rep
    R = B - A @ X
    be = (R.abs().amax(0) / (A.abs().sum(1).amax() * X.abs().amax(0) + B.abs().amax(0))).max()
    assert float(be) <= 1.1e-13  # the default tolerance, plus the check's own rounding


def _potrf(gpu_lla, torch, A, ld=None):
    """FAST device factor of A in a buffer of leading dimension ld (column-major)."""
    n = A.shape[0]
    ld = ld or n
    buf = torch.full((n, ld), -7.0, dtype=A.dtype, device="cuda")
    buf[:, :n] = A.T
    L = buf.T[:n]
    info = gpu_lla.potrf_device(L, algo=gpu_lla.ALGO_FAST)
    torch.cuda.synchronize()
    assert ld == n or bool((buf[:, n:] == -7.0).all()), "rows below the matrix were written"
    return L, int(info.item())


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 128, 129, 192, 193, 257, 320, 1000])
@pytest.mark.parametrize("pad", [0, 3])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_fast_factor(gpu_lla, n, pad, dtype):
    """Digit-sliced trailing updates: edges of the 64-column panels, the 128-row
    tiles and the pairs of panels, against ||L L^T - A|| <= 10 n eps ||A||; the
    upper triangle stays untouched."""
    torch = _torch()
    A, g = _spd(torch, n, 0.5, n)
    d = torch.exp2(20 * torch.rand(n, dtype=torch.float64, device="cuda", generator=g) - 10)
    A = (A * d[:, None] * d[None, :]).to(getattr(torch, dtype))
    A = torch.tril(A) + torch.tril(A, -1).T
    L, info = _potrf(gpu_lla, torch, A, n + pad)
    assert info == -1
    low = torch.tril(L).double()
    S = A.double() / d[:, None] / d[None, :]
    R = (low @ low.T) / d[:, None] / d[None, :] - S
    assert float(R.norm() / S.norm()) <= 10 * n * torch.finfo(A.dtype).eps
    assert bool((torch.triu(L, 1) == torch.triu(A, 1)).all())


@pytest.mark.parametrize("row", [0, 1, 30, 31, 32, 33, 63, 64, 65, 100, 127, 128, 200, 255, 299])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_fast_factor_reports_the_failing_row(gpu_lla, row, dtype):
    torch = _torch()
    A, _ = _spd(torch, 300, 1.0, 3)
    A = A.to(getattr(torch, dtype))
    A[row, row] = -1.0
    L, info = _potrf(gpu_lla, torch, A)
    assert info == row
    if row:
        R = torch.linalg.cholesky(A[:row, :row].double())
        assert float((torch.tril(L[:row, :row]) - R).norm() / R.norm()) <= 10 * 300 * torch.finfo(A.dtype).eps


def test_fast_fp64_factor_non_finite_and_subnormal_rows(gpu_lla):
    """A row without digits (NaN) spoils what a FMA factorisation would spoil and nothing else;
    a subnormal pivot is a pivot."""
    torch = _torch()
    n, bad = 300, 170
    A, _ = _spd(torch, n, 1.0, 5)
    R = torch.linalg.cholesky(A)
    A[bad, 3] = A[3, bad] = float("nan")
    L, info = _potrf(gpu_lla, torch, A)
    assert info == -1
    ok = torch.ones(n, n, dtype=torch.bool, device="cuda").tril()
    ok[bad, 3:] = False
    ok[bad + 1:, bad:] = False
    assert float((L - R)[ok].abs().max()) <= 1e-13
    assert bool(torch.isnan(L[bad, 3:bad + 1]).all()) and bool(torch.isnan(torch.diagonal(L)[bad:]).all())
    D = torch.eye(130, dtype=torch.float64, device="cuda")
    D[70, 70] = 4.0e-310
    L, info = _potrf(gpu_lla, torch, D)
    assert info == -1 and abs(float(L[70, 70]) - 2.0e-155) <= 1e-168 and float(L[129, 129]) == 1.0


def test_fast_fp64_factor_on_two_streams_and_in_a_graph(gpu_lla):
    """Concurrent factorisations of one thread, and replays of a captured one, share no scratch."""
    torch = _torch()
    n = 700
    mats = [_spd(torch, n, 1.0, 20 + i)[0] for i in range(4)]
    want = [_potrf(gpu_lla, torch, A)[0].clone() for A in mats]
    streams = [torch.cuda.Stream() for _ in range(2)]
    out = [A.clone().T for A in mats]
    infos = [torch.empty(1, dtype=torch.int64, device="cuda") for _ in mats]
    torch.cuda.synchronize()
    for i, (L, f) in enumerate(zip(out, infos)):
        gpu_lla.potrf_device(L, algo=gpu_lla.ALGO_FAST, info=f, stream=streams[i % 2])
    torch.cuda.synchronize()
    for L, w, f in zip(out, want, infos):
        assert int(f.item()) == -1 and bool((L == w).all())
    L = mats[0].clone().T
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        gpu_lla.potrf_device(L, algo=gpu_lla.ALGO_FAST, info=infos[0], stream=torch.cuda.current_stream())
    other = mats[1].clone().T
    for i in (1, 2):
        L.copy_(mats[i].T)
        torch.cuda.synchronize()
        graph.replay()
        gpu_lla.potrf_device(other, algo=gpu_lla.ALGO_FAST, info=infos[1], stream=streams[1])
        torch.cuda.synchronize()
        assert bool((L == want[i]).all())
        assert i != 1 or bool((other == want[1]).all())


def _tri(n, dtype, seed, scale):
    """Well-conditioned lower triangle, rows scaled by 2^U(-scale, scale)."""
    rng = np.random.default_rng(seed)
    t = np.tril(rng.standard_normal((n, n)) / np.sqrt(n), -1) + np.diag(rng.uniform(1, 2, n) * rng.choice((-1, 1), n))
    d = np.exp2(np.round(rng.uniform(-scale, scale, n)))
    return (t * d[:, None]).astype(dtype), d


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,m", [(1, 1), (31, 3), (32, 4), (33, 5), (65, 9), (257, 2)])
@pytest.mark.parametrize("scale", [0, 60, 600])
def test_fast_substitution_forms(gpu_lla, dtype, n, m, scale):
    """FAST triangular solves in both directions, with row scales inside and outside the
    range in which rows are divided by their diagonal beforehand: scaling the rows of T and
    of B by powers of two changes nothing."""
    torch = _torch()
    if scale > 60 and dtype == np.float32:
        pytest.skip("outside the type's exponent range")
    t, d = _tri(n, dtype, n + m, scale)
    b0 = np.random.default_rng(m).standard_normal((n, m))
    eps = np.finfo(dtype).eps
    for trans in (0, 1):
        # trans = 1 solves T^T x = b, where the scales are those of the unknowns
        b = (b0 * d[:, None] if not trans else b0).astype(dtype)
        L = torch.from_numpy(np.ascontiguousarray(t.T)).cuda().T
        X = torch.from_numpy(np.ascontiguousarray(b.T)).cuda().T
        gpu_lla.trsm_device(L, X, trans, algo=gpu_lla.ALGO_FAST)
        gpu_lla.device_status()
        x = X.cpu().numpy().astype(np.float64)
        base = (t.astype(np.float64) / d[:, None])
        y = x * d[:, None] if trans else x
        r = (base.T if trans else base) @ y - b0
        den = np.abs(base).sum(1).max() * np.abs(y).max() + np.abs(b0).max()
        assert np.abs(r).max() <= 10 * max(n, 4) * eps * den


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_exact_division_fallbacks_match_the_oracle(gpu_lla, dtype):
    """Quotients that the integer division does not take (subnormal, overflowing, infinite and
    NaN values, zero diagonals) repeat the block with IEEE division: bit-identical to the oracle."""
    from oracle import oracle as ora
    n, tiny = 70, np.finfo(dtype).tiny
    t, _ = _tri(n, dtype, 9, 0)
    b = np.random.default_rng(1).standard_normal((n, 6)).astype(dtype)
    b[:, 1] *= tiny
    b[:, 2] = 0
    b[5, 2] = -0.0
    b[:, 3] *= np.finfo(dtype).max / 8
    b[40, 4] = np.inf
    b[41, 5] = np.nan
    with np.errstate(all="ignore"):
        for k, v in ((None, 0), (33, 0.0), (50, tiny / 4), (66, np.inf)):
            tt = t.copy()
            if k is not None:
                tt[k, k] = v
            want, got = b.copy(), b.copy()
            ora.solve_triangular_inplace(tt, want, "lower")
            prev = gpu_lla.set_algorithm(gpu_lla.ALGO_EXACT)
            try:
                gpu_lla.solve_triangular_inplace(tt, got, "lower")
            finally:
                gpu_lla.set_algorithm(prev)
            same = (got == want) | (np.isnan(got) & np.isnan(want))
            assert same.all() and (np.signbit(got) == np.signbit(want))[~np.isnan(want)].all(), (k, v)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 64, 65, 97])
@pytest.mark.parametrize("kind", ["plain", "fails", "tiny", "inf", "nan"])
def test_exact_factor_matches_the_oracle(gpu_lla, dtype, n, kind):
    """EXACT factor at the edges of its 32-column panels and 16-row tiles, also where integer roots
    and quotients do not apply (subnormal values, infinities, NaN) and at failing pivots."""
    from oracle import oracle as ora
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, n))
    a = (g @ g.T / n + np.eye(n)).astype(dtype)
    k = int(rng.integers(0, n))
    if kind == "fails":
        a[k, k] = -a[k, k]
    elif kind == "tiny":
        a[k] *= np.finfo(dtype).tiny
        a[:, k] = a[k]
        a[k, k] = np.finfo(dtype).tiny / 8
    elif kind == "inf":
        a[k, k] = np.inf
    elif kind == "nan":
        a[k, k // 2] = np.nan
    want, got = a.copy(), a.copy()
    with np.errstate(all="ignore"):
        st = ora.cholesky_inplace_dirty(want)
    prev = gpu_lla.set_algorithm(gpu_lla.ALGO_EXACT)
    try:
        fail = -1
        try:
            gpu_lla.cholesky_inplace_dirty(got)
        except gpu_lla.NotPositiveDefinite as e:
            fail = e.index
    finally:
        gpu_lla.set_algorithm(prev)
    assert (fail >= 0) == (st["code"] != 0) and (fail < 0 or fail == st["index"])
    assert ((got == want) | (np.isnan(got) & np.isnan(want))).all()


@pytest.mark.parametrize("n", [1, 33, 64, 65, 200, 1000])
@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32, 33, 65])
def test_fp64_residual_tiles(gpu_lla, n, m):
    """FP64 residual on each of its tile widths, against an FP64 product of the same operands:
    two sums of n products in different orders differ by at most 2 n eps |A| |x|."""
    torch = _torch()
    A, g = _spd(torch, n, 1.0, n + m)
    X = torch.randn(m, n, dtype=torch.float64, device="cuda", generator=g).T
    B = torch.randn(m, n, dtype=torch.float64, device="cuda", generator=g).T
    R = torch.empty(m, n, dtype=torch.float64, device="cuda").T
    low = torch.tril(A).T.contiguous().T  # only the lower triangle is read
    gpu_lla.residual_device(low, X, B, R, "fp64")
    torch.cuda.synchronize()
    tol = 2 * (n + 2) * 2.2e-16 * (A.abs() @ X.abs() + B.abs())
    assert bool(((R - (B - A @ X)).abs() <= tol).all())


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("k", [1, 2, 15, 16, 17, 32, 33, 45, 48, 49, 63, 64, 80])
@pytest.mark.parametrize("n", [100, 129, 5000])
def test_cholesky_qr_forms(gpu_lla, dtype, k, n):
    """Gram products dealt out one by one or in tiles, and substitutions row by row or through
    the transposed block: L against the Gram matrix (n products summed in any order: n eps
    sum |v||v|, plus the factor's k eps), U bit-identical to the oracle's solve with that L."""
    from oracle import oracle as ora
    rng = np.random.default_rng(k + n)
    v = np.asfortranarray((rng.standard_normal((n, k)) * 10.0 ** rng.uniform(-1, 1, k)).astype(dtype))
    u, l = gpu_lla.orthonormalize(v)
    w = v.astype(np.float64)
    low = l.astype(np.float64)
    err = np.abs(low @ low.T - w.T @ w)
    norms = np.sqrt((w * w).sum(0))
    assert (err <= (n + 2 * k + 2) * np.finfo(dtype).eps * norms[:, None] * norms[None, :]).all()
    vt = np.array(v.T, order="C")
    assert ora.solve_triangular_inplace(np.array(l, order="C"), vt, "lower")["code"] == 0
    assert np.array_equal(u, vt.T)
    y = np.asfortranarray(rng.standard_normal((n, 7)).astype(dtype))
    lyy = np.linalg.cholesky((y.astype(np.float64).T @ y.astype(np.float64))).astype(dtype)
    x = v.copy()
    gpu_lla.apply_constraints(x, lyy, y)
    g = y.astype(np.float64).T @ w
    want = w - y.astype(np.float64) @ np.linalg.solve(lyy.astype(np.float64), g)
    assert np.abs(x - want).max() <= 1e3 * np.finfo(dtype).eps * np.sqrt(n) * np.abs(w).max()


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(4, 128), (2, 256), (1, 128)])
def test_batch_orders_and_failures(gpu_lla, dtype, shape):
    """Every order around the blocks, tiles and panel forms, 0-8 right-hand sides, with failing and
    NaN systems among them: residuals within 10 n eps, first failing rows, untouched upper parts,
    and B left alone where the factorisation fails."""
    torch = _torch()
    orders = [1, 2, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32, 33, 40, 47, 48, 49, 63, 64, 65, 95, 96, 97, 127, 128, 129,
              160, 191, 192, 193, 223, 224, 225, 239, 240, 241, 254, 255, 256]
    rng = np.random.default_rng(1)
    n = np.array(orders * 3, dtype=np.int32)
    m = np.array([(7 * i) % 9 for i in range(len(n))], dtype=np.int32)
    bad = {i: int(rng.integers(0, n[i])) for i in range(len(orders), 2 * len(orders))}
    nan = set(range(2 * len(orders), len(n), 5))
    As, Bs = [], []
    for i, k in enumerate(n):
        g = rng.standard_normal((k, k))
        a = g @ g.T / k + 0.5 * np.eye(k)
        if i in bad:
            a[bad[i], bad[i]] = -1.0
        if i in nan:
            a[k // 2, k // 3] = np.nan
        As.append(a)
        Bs.append(rng.standard_normal((k, m[i])))
    plan = gpu_lla.BatchPlan(n, m, dtype)
    plan.set_shape(*shape)
    ap, bp = plan.pack(As, Bs)
    A, B = torch.from_numpy(ap.copy()).cuda(), torch.from_numpy(bp.copy()).cuda()
    info = torch.empty(len(n), dtype=torch.int32, device="cuda")
    plan.solve(A, B, info)
    torch.cuda.synchronize()
    X, info, out = plan.unpack_x(B.cpu().numpy()), info.cpu().numpy(), A.cpu().numpy()
    eps = np.finfo(plan.np_dtype).eps
    b0 = plan.unpack_x(bp)
    for i, k in enumerate(n):
        fac = out[plan.a_off[i]:plan.a_off[i] + k * k].reshape((k, k), order="F")
        a = ap[plan.a_off[i]:plan.a_off[i] + k * k].reshape((k, k), order="F")
        up = np.triu(np.ones((k, k), bool), 1)
        assert ((fac == a) | (np.isnan(fac) & np.isnan(a)))[up].all(), i
        if i in bad:
            assert info[i] == bad[i] and (X[i] == b0[i]).all(), (i, k)
            continue
        assert info[i] == -1, (i, k, info[i])
        if i in nan:
            continue
        ad, x = a.astype(np.float64), X[i].astype(np.float64)
        low = np.tril(fac).astype(np.float64)
        assert np.abs(low @ low.T - ad).max() <= 10 * max(k, 4) * eps * np.abs(ad).sum(1).max(), (i, k)
        r = np.abs(ad @ x - b0[i])
        if x.size:
            den = np.abs(ad).sum(1).max() * np.abs(x).max(0) + np.abs(b0[i]).max(0)
            assert (r.max(0) <= 10 * max(k, 4) * eps * den).all(), (i, k)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 65, 96, 97, 127, 128, 129, 160, 255, 257, 385])
@pytest.mark.parametrize("pad", [0, 4, 3])
def test_mixed_factor_blocks(gpu_lla, n, pad):
    """The mixed solve's diagonal blocks: edges of the 32-column steps and the 128-column blocks,
    16-byte aligned columns and not: ||L L^T - A|| <= 10 n eps ||A||, nothing else written, and a
    negative pivot reported in its block."""
    torch = _torch()
    A, _ = _spd(torch, n, 0.5, n)
    A = A.float()
    for row in (None, n - 1):
        M = A.clone()
        if row is not None:
            M[row, row] = -1.0
        buf = torch.full((n, n + pad), -7.0, dtype=torch.float32, device="cuda")
        buf[:, :n] = M.T
        L = buf.T[:n]
        info = gpu_lla.spotrf_mixed_device(L, update="bf16x6")
        torch.cuda.synchronize()
        assert bool((buf[:, n:] == -7.0).all())
        if row is not None:
            assert int(info.item()) == row // 128 * 128
            continue
        assert int(info.item()) == -1
        low = torch.tril(L).double()
        assert float((low @ low.T - A.double()).norm() / A.double().norm()) <= 10 * n * torch.finfo(torch.float32).eps
