"""Host code of the library on a CUDA runtime without a GPU (tests/fake_cuda.cpp): what the
entry points ask of the runtime, on two devices."""
import ctypes
import glob
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "linfa-linalg_gb300")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    objs = sorted(glob.glob(os.path.join(PKG, "_build", "*.o")))
    if not objs or not shutil.which("g++"):
        pytest.skip("the library's objects are built by build()")
    so = str(tmp_path_factory.mktemp("fake") / "liblla_fake.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-I", os.path.join(CUDA, "include"), "-o", so,
                    os.path.join(ROOT, "tests", "fake_cuda.cpp")] + objs +
                   ["-Wl,-Bsymbolic", "-Wl,--no-undefined", "-lpthread", "-ldl", "-lm"], check=True)
    lib = ctypes.CDLL(so)
    lib.fake_log.restype = ctypes.c_char_p
    return lib


@pytest.fixture(autouse=True)
def own_cache(tmp_path, monkeypatch):
    """An autotune cache file of the test's own."""
    monkeypatch.setenv("LLA_AUTOTUNE_CACHE", str(tmp_path / "autotune.txt"))
    return tmp_path / "autotune.txt"


def on_device(lib, dev, fn):
    """fn() on a host thread of its own, bound to a device: its result."""
    out = []

    def body():
        lib.fake_set_device(dev)
        out.append(fn())

    t = threading.Thread(target=body)
    t.start()
    t.join()
    return out[0]


def _plan(lib, refined=False):
    n, m = np.full(40, 16, np.int32), np.ones(40, np.int32)
    plan = P()
    assert lib.lla_batch_plan_create(I64(40), P(n.ctypes.data), P(m.ctypes.data), 8, ctypes.byref(plan), None) == 0
    if refined:
        assert lib.lla_batch_set_refined(plan, 1, None) == 0
    return plan


def _shape(lib, plan):
    c, t = ctypes.c_int(), ctypes.c_int()
    assert lib.lla_batch_plan_info(plan, None, None, None, None, ctypes.byref(c), ctypes.byref(t), None) == 0
    return c.value, t.value


def _autotune(lib, plan):
    a, b, info = np.zeros((40, 256)), np.zeros((40, 16)), np.zeros(40, np.int32)
    assert lib.lla_batch_autotune(plan, P(a.ctypes.data), P(b.ctypes.data), P(info.ctypes.data), None, None, None) == 0


I64, P = ctypes.c_int64, ctypes.c_void_p


def _launches(lib, dev, kernel):
    """Grid sizes of the launches of a kernel on a device since the last clear."""
    rows = [r.split(" ", 2) for r in lib.fake_log().decode().splitlines()]
    return [int(g) for d, g, name in rows if int(d) == dev and kernel in name]


def _fast_factor(lib, fn, dtype):
    a, info = np.eye(512, dtype=dtype), np.zeros(1, np.int64)
    return fn(P(a.ctypes.data), I64(512), I64(512), 2, P(info.ctypes.data), None, None)


def _batch(lib, elem, refined):
    n, m = np.full(40, 16, np.int32), np.ones(40, np.int32)
    plan = P()
    assert lib.lla_batch_plan_create(I64(40), P(n.ctypes.data), P(m.ctypes.data), elem, ctypes.byref(plan), None) == 0
    if refined:
        st = lib.lla_batch_set_refined(plan, 1, None)
        if st:
            return st
    a, b, info = np.zeros((40, 256)), np.zeros((40, 16)), np.zeros(40, np.int32)
    fn = lib.lla_dbatch_posv_device if elem == 8 else lib.lla_sbatch_posv_device
    st = fn(plan, P(a.ctypes.data), P(b.ctypes.data), P(info.ctypes.data), None, None)
    lib.lla_batch_plan_destroy(plan)
    return st


def _residual(lib, method):
    n, m = 300, 8
    a, x, b, r = np.zeros((n, n)), np.zeros((m, n)), np.zeros((m, n)), np.zeros((m, n))
    p = [P(v.ctypes.data) for v in (a, x, b, r)]
    return lib.lla_dresidual_device(p[0], I64(n), I64(n), p[1], I64(n), p[2], I64(n), p[3], I64(n), I64(m), method,
                                    None, None)


# entry point, kernel with more than 48 KiB of dynamic shared memory (or a grid by the
# multiprocessor count), and whether a multiprocessor holds several of its CTAs
CALLS = {
    "factor f64": (lambda lib: _fast_factor(lib, lib.lla_dpotrf_device, np.float64), "fc_update_kernel", 1),
    "factor f32": (lambda lib: _fast_factor(lib, lib.lla_spotrf_device, np.float32), "fc_update_kernel", 1),
    "batch f64": (lambda lib: _batch(lib, 8, False), "batch_posv_kernel", 4),
    "batch f32": (lambda lib: _batch(lib, 4, False), "batch_posv_kernel", 4),
    "batch refined": (lambda lib: _batch(lib, 8, True), "batch_posv_refined_kernel", 2),
    "residual by slices": (lambda lib: _residual(lib, 1), "oz_residual_kernel", None),
}


@pytest.mark.parametrize("call", CALLS)
def test_a_second_device_is_asked_for_itself(fake, call):
    """Kernel attributes and multiprocessor counts belong to a device: the same call from threads
    bound to two devices is launched on both, with each device's own grid."""
    run, kernel, per_sm = CALLS[call]
    for dev, sms in ((0, 5), (1, 7), (0, 5)):
        fake.fake_clear()
        assert on_device(fake, dev, lambda: run(fake)) == 0, f"refused on device {dev}"
        grids = _launches(fake, dev, kernel)
        assert grids and (per_sm is None or max(grids) == min(per_sm * sms, 40)), grids


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_a_captured_factor_allocates_beside_the_graph(fake, dtype):
    """A captured FAST factor puts no allocation into the caller's graph, whose copies could not
    run otherwise; the graph keeps the scratch, and once it is gone the next call frees it."""
    fn = fake.lla_dpotrf_device if dtype == np.float64 else fake.lla_spotrf_device
    a, info = np.eye(300, dtype=dtype), np.zeros(1, np.int64)

    def factor(stream):
        return fn(P(a.ctypes.data), I64(300), I64(300), 2, P(info.ctypes.data), stream, None)

    def body():
        stream, graph = P(), P()
        fake.cudaStreamCreateWithFlags(ctypes.byref(stream), 1)
        assert factor(stream) == 0  # creates the thread's workspace
        blocks, nodes = fake.fake_pool_blocks(), fake.fake_alloc_nodes()
        fake.cudaStreamBeginCapture(stream, 1)
        assert factor(stream) == 0
        fake.cudaStreamEndCapture(stream, ctypes.byref(graph))
        assert fake.fake_alloc_nodes() == nodes
        assert factor(stream) == 0 and fake.fake_pool_blocks() == blocks + 1  # the graph's
        fake.cudaGraphDestroy(graph)
        assert factor(stream) == 0 and fake.fake_pool_blocks() == blocks
        return True

    assert on_device(fake, 0, body)


def test_shapes_tuned_for_other_kernels_are_not_taken(fake, own_cache):
    """Cache entries without this generation's mark leave the default shape; its own are taken up."""
    key = "b8:c40:h40-0-0-0-0-0-0-0-0:m1"
    own_cache.write_text(f"{key} 2 256\nk1:{key} 2 256\n{key}:r 1 128\n")
    assert _shape(fake, _plan(fake)) == (4, 128) and _shape(fake, _plan(fake, True)) == (2, 256)
    tuned = _plan(fake)
    _autotune(fake, tuned)  # (every candidate takes the same time here: the first stays)
    assert _shape(fake, tuned) == (1, 256) == _shape(fake, _plan(fake))


def test_a_shape_tuned_for_one_mode_stays_with_it(fake):
    """Switching the mode takes that mode's tuned shape or its default, not the other mode's; a
    shape that the caller set stays."""
    plan = _plan(fake)
    _autotune(fake, plan)
    assert _shape(fake, plan) == (1, 256)
    assert fake.lla_batch_set_refined(plan, 1, None) == 0 and _shape(fake, plan) == (2, 256)
    assert fake.lla_batch_set_refined(plan, 0, None) == 0 and _shape(fake, plan) == (1, 256)
    assert _shape(fake, _plan(fake, True)) == (2, 256)  # a plan that found the plain shape in the cache
    own = _plan(fake)
    assert fake.lla_batch_set_shape(own, 3, 128) == 0
    assert fake.lla_batch_set_refined(own, 1, None) == 0 and _shape(fake, own) == (3, 128)


@pytest.mark.parametrize("dtype,n,k,rows", [
    (np.float64, 100, 24, True), (np.float64, 600, 32, False), (np.float64, 2559, 32, False), (np.float64, 2560, 32, True),
    (np.float64, 3839, 48, False), (np.float64, 3840, 48, True), (np.float64, 60000, 49, False),
    (np.float32, 100, 48, True), (np.float32, 60000, 49, False)])
def test_cholesky_qr_rows_or_substitution(fake, dtype, n, k, rows):
    """Short blocks of many FP64 columns go through the substitution kernel."""
    v, u, low = np.zeros((n, k), dtype), np.zeros((n, k), dtype), np.zeros((k, k), dtype)
    fn = fake.lla_dorthonormalize if dtype == np.float64 else fake.lla_sorthonormalize

    def body():
        fake.fake_clear()
        views = [x for m in (v, u, low) for x in (P(m.ctypes.data), I64(len(m)), I64(k), I64(k), I64(1))]
        return fn(*views, None)

    assert on_device(fake, 0, body) == 0
    assert bool(_launches(fake, 0, "solve_rows_kernel")) == rows and bool(_launches(fake, 0, "trsm_lookback")) != rows
