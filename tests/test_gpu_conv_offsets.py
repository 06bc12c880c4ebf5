"""Conv windows at any element of their arena: the forms that read rows by vector (exact and chunked prefill, chunked verify) give
for windows that start 2, 4 and 6 bytes past an aligned place the bits they give for aligned ones."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.fixture(scope="module")
def K():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return importlib.import_module("glm53f-afd_b200.kernel")


# Lengths shorter than the window (1, 2: rows of several taps come from it) and of one pass and more.
@pytest.mark.parametrize("what, lens", [("exact", [1, 17, 2]), ("exact", [40, 8]), ("chunked", [1, 70, 2]), ("chunked", [3]), ("verify", [1, 2, 7, 16])])
def test_windows_at_unaligned_offsets(K, what, lens):
    h, n, total = 2, len(lens), sum(lens)
    g = torch.Generator(device="cuda").manual_seed(total)
    c, width = K.channels(h), h * DK
    stride, per = c + 8, 3 * c + 8  # a window and a gap
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=g) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
    w = K.Weights(h, buf(rn(c * 4, 0.5)), buf(rn(h, 0.5, torch.float32)), buf(rn(width, 1.0, torch.float32)), buf(1 + rn(DK, 0.1)), 1e-5, -5.0)
    p, gates, windows = rn(total * stride), rn(total * 2 * width), rn(n * 3 * c).view(n, 3 * c)
    states = rn(n * K.state_len(h), 0.3, torch.bfloat16)
    stream, got = K.Stream(), []
    for shift in range(4):
        conv = torch.zeros(n, per, dtype=torch.bfloat16, device="cuda")
        conv[:, shift:shift + 3 * c] = windows
        st, out = states.clone(), torch.zeros(total * width, dtype=torch.bfloat16, device="cuda")
        meta = K.BatchMeta.new(n)
        meta.set([K.Request(r, i * per + shift, i * K.state_len(h)) for i, r in enumerate(lens)])
        rows = (K.RowView.dense(buf(p), stride), c, K.RowView.new(buf(gates), 0, 2 * width), K.RowView.new(buf(gates), width, 2 * width))
        view, saves = K.RowView.dense(buf(out), width), None
        if what == "verify":
            before = K.set_verify_form(K.Form.CHUNKED)
            saves = K.Saves.alloc(h, total)
            call = K.ChainBatch(w, *rows, buf(conv.view(-1)), buf(st), K.StateOut.Skip, view, saves)
        else:
            before = K.set_prefill_form(K.Form.CHUNKED if what == "chunked" else K.Form.EXACT)
            call = K.PrefillBatch(w, *rows, buf(conv.view(-1)), buf(st), K.StateOut.InPlace, view, 0, K.PrefillWorkspace.new(h, n, 64))
        try:
            call.launch_bf16_state(meta, stream)
            torch.cuda.synchronize()
        finally:
            (K.set_verify_form if what == "verify" else K.set_prefill_form)(before)
        kept = [] if saves is None else [b.t.clone() for b in (saves.k, saves.v, saves.g, saves.b)]
        assert not conv[:, :shift].any() and not conv[:, shift + 3 * c:].any()  # nothing is written beside the windows
        got.append([out, st, conv[:, shift:shift + 3 * c].contiguous(), *kept])
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
