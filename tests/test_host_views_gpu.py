"""Host calls whose factorisation fails, or has to be repeated in the reference's order,
with the work that was enqueued behind it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spd(n, dtype=np.float64):
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, n))
    return (g @ g.T / n + np.eye(n)).astype(dtype)


def _ms(gpu_lla, fn):
    """Milliseconds of the substitutions of one call."""
    gpu_lla.profile_start()
    try:
        fn()
    except gpu_lla.NotPositiveDefinite:
        pass
    return gpu_lla.profile_stop()["trsm"][0]


@pytest.mark.parametrize("call", ["solvec", "invc"])
@pytest.mark.parametrize("n", [600, 1500])
def test_a_failed_factor_costs_no_substitution(gpu_lla, call, n):
    """The substitutions enqueued behind a factor that fails return at once: under a quarter of
    what they take behind one that stands (launches of empty blocks against dependent row blocks)."""
    a, b = _spd(n), np.ones((n, 4))
    bad = a.copy()
    bad[n - 1, n - 1] = -1.0

    def run(m):
        m = m.copy()
        return gpu_lla.solvec_inplace(m, b.copy()) if call == "solvec" else gpu_lla.invc_inplace(m)

    run(a)
    good = min(_ms(gpu_lla, lambda: run(a)) for _ in range(3))
    assert min(_ms(gpu_lla, lambda: run(bad)) for _ in range(3)) < good / 4


@pytest.mark.parametrize("n", [700, 1100])
@pytest.mark.parametrize("layout", ["C", "F", "strided"])
@pytest.mark.parametrize("kind", ["fails", "near singular"])
def test_outcomes_that_are_not_the_usual_one(gpu_lla, n, layout, kind):
    """A failing factor leaves B alone and in A what the EXACT order leaves; a FAST factor with a tiny
    pivot is repeated in EXACT order, and the solution belongs to that factor."""
    a = _spd(n)
    if kind == "fails":
        a[n // 2, n // 2] = -1.0
    else:
        a[n - 1] *= 1e-9  # a last pivot of about 1e-14 of the diagonal
        a[:, n - 1] *= 1e-9
        row = np.linalg.solve(a[:n - 1, :n - 1], a[:n - 1, n - 1])
        a[n - 1, n - 1] = a[:n - 1, n - 1] @ row * (1 + 1e-12)
    b = np.random.default_rng(1).standard_normal((n, 3))

    def views():
        out = []
        for v in (a, b):
            if layout == "strided":
                big = np.full((2 * v.shape[0], 2 * v.shape[1]), 7.0)
                w = big[::2, ::2]
            else:
                w = np.empty(v.shape, order=layout)
            w[...] = v
            out.append(w)
        return out

    def run(algo):
        va, vb = views()
        prev = gpu_lla.set_algorithm(algo)
        try:
            fail = -1
            try:
                gpu_lla.solvec_inplace(va, vb)
            except gpu_lla.NotPositiveDefinite as e:
                fail = e.index
        finally:
            gpu_lla.set_algorithm(prev)
        return va, vb, fail

    ea, eb, ef = run(gpu_lla.ALGO_EXACT)
    fa, fb, ff = run(gpu_lla.ALGO_FAST)
    assert ef == ff == (n // 2 if kind == "fails" else ff)
    assert (ea == fa).all()
    assert (np.triu(fa, 1) == np.triu(a, 1)).all()
    if ff >= 0:
        assert (eb == b).all() and (fb == b).all()
    else:
        low = np.tril(fa)
        for x in (eb, fb):
            r = np.abs(low @ (low.T @ x) - b)
            assert (r <= 10 * n * 2.3e-16 * (np.abs(low) @ (np.abs(low.T) @ np.abs(x)) + np.abs(b))).all()
