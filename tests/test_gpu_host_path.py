"""The native host path and what it uploads by: words carried in kernel parameters at the edges of a launch's capacity,
page lists in parameters against page lists on the device, and the launches it must leave to the Python checks."""
import ctypes as C
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 255, 257, 999, 1000, 1001, 2500])
def test_store_words(pkg, n):
    lib = pkg.ffi.load()
    host = np.random.default_rng(n).integers(0, 1 << 32, max(n, 1), dtype=np.uint32)
    dst = torch.zeros(n + 4, dtype=torch.int32, device="cuda")
    assert lib.glm53f_kda_store_words(dst.data_ptr(), host.ctypes.data, n, torch.cuda.current_stream().cuda_stream) == 0
    got = dst.cpu().numpy().view(np.uint32)
    assert (got[:n] == host[:n]).all() and not got[n:].any()


@pytest.mark.parametrize("n_pages", [1, 899, 900])
@pytest.mark.parametrize("save", [1, 0])
def test_mark_copy_with_the_page_list_in_the_parameters(pkg, n_pages, save):
    lib = pkg.ffi.load()
    pb, rng = 1024, np.random.default_rng(n_pages)
    pages = np.sort(rng.permutation(n_pages + 5)[:n_pages]).astype(np.int32)
    size = n_pages * pb - 16 * (n_pages > 1)  # a last page that is not full
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    sizes = (C.c_int64 * 3)(size, 0, 0)
    both = []
    for inline in (False, True):
        g = torch.Generator(device="cuda").manual_seed(3)
        pool = torch.randint(0, 256, ((n_pages + 5) * pb,), dtype=torch.uint8, device="cuda", generator=g)
        part = torch.randint(0, 256, (size,), dtype=torch.uint8, device="cuda", generator=g)
        parts = (C.c_void_p * 3)(part.data_ptr(), None, None)
        if inline:
            assert lib.glm53f_kda_mark_copy_list(pool.data_ptr(), pb, pages.ctypes.data, n_pages, parts, sizes, save, stream) == 0
        else:
            d = torch.from_numpy(pages).cuda()
            assert lib.glm53f_kda_mark_copy(pool.data_ptr(), pb, d.data_ptr(), parts, sizes, save, stream) == 0
        both.append((pool.cpu(), part.cpu()))
    assert torch.equal(both[0][0], both[1][0]) and torch.equal(both[0][1], both[1][1])
    # a list of another length, or one too long for the parameters, is rejected before anything runs
    assert lib.glm53f_kda_mark_copy_list(pool.data_ptr(), pb, pages.ctypes.data, n_pages - 1, parts, sizes, save, stream) == 1
    assert lib.glm53f_kda_mark_copy_list(pool.data_ptr(), pb, pages.ctypes.data, 901, parts, sizes, save, stream) == 1


def test_calls_with_an_error_keep_their_errors(pkg):
    core, h = importlib.import_module("glm53f-afd_b200.core"), 2
    z = lambda n, d: torch.zeros(n, dtype=d, device="cuda")
    cu, off = torch.tensor([0, 1], dtype=torch.int32, device="cuda"), z(1, torch.int64)
    ok = dict(heads=h, rows=1, cu_rows=cu, q=z(h * 128, torch.bfloat16), k=z(h * 128, torch.bfloat16), v=z(h * 128, torch.bfloat16),
              g=z(h * 128, torch.float32), beta=z(h, torch.float32), state=z(h * 128 * 128, torch.float32), state_off=off,
              out=z(h * 128, torch.bfloat16))
    core.decode_batch(**ok)
    for bad, text in ((dict(q=z(h * 128 - 1, torch.bfloat16)), "q holds"), (dict(g=z(h * 128, torch.float64)), "g has dtype"), (dict(out=None), "rejected"),
                      (dict(v=z(h * 128, torch.bfloat16).cpu()), "v must be"), (dict(flags=64), "rejected"), (dict(max_state_off=1), "exceeds")):
        with pytest.raises(core.Invalid, match=text):
            core.decode_batch(**{**ok, **bad})
    torch.cuda.synchronize()
    assert core.device_status() == 0


BIG = 1 << 62


@pytest.mark.parametrize("what, text", [
    (dict(conv_offset=(1 << 63) - 1), "conv: elements"), (dict(state_offset=(1 << 63) - 8), "state: elements"), (dict(conv_offset=-1), "conv: elements"),
    (dict(b_off=(1 << 63) - 1), "p"), (dict(rows=2, p_stride=BIG), "p"), (dict(p_stride=BIG), "p"), (dict(a_stride=BIG), "a"), (dict(g_stride=3 * BIG // 2), "g"), (dict(p_offset=(1 << 63) - 4), "p"),
    (dict(out_stride=255), "out"), (dict(state_offset=1), "state: "), (dict(rows=3), "p"), (dict(saves=1), "saves hold")])
def test_a_chain_call_with_an_error_keeps_its_error(pkg, what, text):
    """Extents that 64 bits cannot hold among them: the checks on the native path may not wrap."""
    K = importlib.import_module("glm53f-afd_b200.kernel")
    h, rows, n = 2, 2, 2
    c, width = K.channels(h), h * 128
    buf = lambda elems, size=2: K.DeviceBuffer(torch.zeros(elems * size, dtype=torch.uint8, device="cuda"))
    w = K.Weights(h, buf(c * 4), buf(h, 4), buf(width, 4), buf(128), 1e-5, -5.0)
    meta = K.BatchMeta.new(n)

    def call(conv_offset=0, state_offset=K.state_len(h), b_off=c, p_stride=c + h, a_stride=width, g_stride=width, out_stride=width, p_offset=0, rows=1, saves=0):
        meta.set([K.Request(rows, 0, 0), K.Request(1, conv_offset, state_offset)])
        K.ChainBatch(w, K.RowView.new(buf(2 * (c + h)), p_offset, p_stride), b_off, K.RowView.new(buf(2 * width), 0, a_stride), K.RowView.new(buf(2 * width), 0, g_stride),
                     buf(3 * c), buf(n * K.state_len(h), 4), K.StateOut.InPlace, K.RowView.new(buf(2 * width), 0, out_stride),
                     K.Saves.alloc(h, saves) if saves else None).launch(meta, K.Stream())

    call()
    with pytest.raises(K.Invalid, match="^" + text):
        call(**what)
    torch.cuda.synchronize()


@pytest.mark.parametrize("entry", ["core", "chain"])
def test_a_blocked_launch_does_not_stop_other_threads(pkg, entry):
    """More launches than the queue holds behind a kernel of 0.6 s: the launch that finds it full blocks, its thread alone."""
    import threading
    import time

    core, K = (importlib.import_module("glm53f-afd_b200." + m) for m in ("core", "kernel"))
    h = 1
    z = lambda n, d=torch.bfloat16: torch.zeros(n, dtype=d, device="cuda")
    if entry == "core":
        cu, off, q, k, v, g, beta = torch.tensor([0, 1], dtype=torch.int32, device="cuda"), z(1, torch.int64), z(128), z(128), z(128), z(128, torch.float32), z(1, torch.float32)
        state, out = z(128 * 128, torch.float32), z(128)
        launch = lambda: core.decode_batch(h, 1, cu, q, k, v, g, beta, state, off, out=out)
    else:
        c, buf = K.channels(h), lambda n, size=2: K.DeviceBuffer(z(n * size, torch.uint8))
        w, meta, s = K.Weights(h, buf(c * 4), buf(h, 4), buf(128, 4), buf(128), 1e-5, -5.0), K.BatchMeta.new(1), K.Stream()
        meta.set([K.Request(1, 0, 0)])
        call = K.ChainBatch(w, K.RowView.dense(buf(c + h), c + h), c, K.RowView.dense(buf(128), 128), K.RowView.dense(buf(128), 128), buf(3 * c),
                            buf(K.state_len(h), 4), K.StateOut.InPlace, K.RowView.dense(buf(128), 128))
        launch = lambda: call.launch(meta, s)
    launch()
    torch.cuda.synchronize()
    gaps, stop = [], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        torch.cuda._sleep(1_100_000_000)
        t0 = time.perf_counter()
        for _ in range(6000):
            launch()
        blocked = time.perf_counter() - t0
    finally:
        stop.set()
        thread.join()
        torch.cuda.synchronize()
    if blocked < 0.4:
        pytest.skip("the queue held every launch")
    assert max(gaps) < 0.15


def test_launches_without_the_native_module(pkg, monkeypatch):
    """The same call through the native path and through the Python checks and ctypes."""
    ffi, K = (importlib.import_module("glm53f-afd_b200." + m) for m in ("ffi", "kernel"))
    h, got = 2, []
    g = torch.Generator(device="cuda").manual_seed(1)
    c, width = K.channels(h), h * 128
    buf = lambda m, s=1.0, d=torch.bfloat16: K.DeviceBuffer((torch.randn(m, device="cuda", generator=g) * s).to(d).view(torch.uint8))
    w = K.Weights(h, buf(c * 4, 0.5), buf(h, 0.5, torch.float32), buf(width, 1.0, torch.float32), buf(128), 1e-5, -5.0)
    p, gates, conv, state, meta = buf(c + h), buf(2 * width), buf(3 * c), buf(K.state_len(h), 0.3, torch.float32), K.BatchMeta.new(1)
    meta.set([K.Request(1, 0, 0)])
    for native in (True, False):
        if not native:
            monkeypatch.setattr(ffi, "_native", ffi._PythonPath)
        st, out = K.DeviceBuffer(state.t.clone()), K.DeviceBuffer.zeroed(2 * width)
        K.ChainBatch(w, K.RowView.dense(p, c + h), c, K.RowView.new(gates, 0, width), K.RowView.new(gates, width, width), conv, st, K.StateOut.InPlace,
                     K.RowView.dense(out, width)).launch(meta, K.Stream())
        torch.cuda.synchronize()
        got.append((out.t, st.t))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and got[0][0].any()


@pytest.mark.parametrize("capacity", [1, 3, 166, 167, 700, 5000])
def test_metadata_in_stream_order(pkg, capacity):
    """BatchMeta.set_on at the edges of what a launch and a few launches carry: the device holds what `set` puts there, and a
    launch queued before still reads what was there then."""
    K = importlib.import_module("glm53f-afd_b200.kernel")
    n = min(capacity, 600)
    first, second = ([K.Request(1 + (i + s) % 3, 8 * i + s, 64 * i + s) for i in range(n)] for s in (0, 5))
    metas = [K.BatchMeta.new(capacity) for _ in range(2)]
    metas[0].set(first)
    metas[1].set(first)
    was = metas[0]._all.t.clone()
    torch.cuda.synchronize()
    torch.cuda._sleep(20_000_000)
    seen = metas[0]._all.t.clone()  # in stream order, ahead of the new metadata
    metas[0].set_on(second, [1] * n, K.Stream())
    metas[1].set(second, [1] * n)
    torch.cuda.synchronize()
    assert torch.equal(seen, was) and torch.equal(metas[0]._all.t, metas[1]._all.t) and was.any()
    assert metas[0]._extent == metas[1]._extent and metas[0].requests() == second
