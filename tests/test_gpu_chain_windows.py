"""The persistent recurrent kernel where a block meets windows of different lengths in turn: single rows (cooked by four warps
together), longer windows (a row per warp), empty ones, more units than blocks so that every ring wraps, and weights that are
not 16-byte aligned.  Each request alone, with aligned weights, must leave the same bits."""
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


@pytest.mark.parametrize("state", ["f32", "bf16"])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("lens", [[1] * 12, [1, 0, 2, 5, 1, 16, 3, 1, 1, 4], [17, 1, 9, 8, 1, 33]])
def test_mixed_windows_have_the_bits_of_single_requests(K, lens, shift, state):
    h, g = 32, torch.Generator(device="cuda").manual_seed(sum(lens) + len(lens))
    c, width, total, n = K.channels(h), h * DK, sum(lens), len(lens)
    stride = c + 64
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=g) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))

    def off(t):  # the same values, `shift` elements into a buffer
        return torch.cat([t[:shift], t])[shift:]

    cw, a_log, dtb, nw = rn(c * 4, 0.5), rn(h, 0.5, torch.float32), rn(width, 1.0, torch.float32), 1 + rn(DK, 0.1)
    p, gates, conv = rn(total * stride), rn(total * 2 * width), rn(n * 3 * c)
    states = rn(n * K.state_len(h), 0.3, torch.bfloat16 if state == "bf16" else torch.float32)

    def run(weights, which):
        st, out = states.clone(), torch.full((total * width,), -1.0, dtype=torch.bfloat16, device="cuda")
        for group in which:
            meta = K.BatchMeta.new(len(group))
            first = sum(lens[:group[0]])
            meta.set([K.Request(lens[i], i * 3 * c, i * K.state_len(h)) for i in group])
            rows = (K.RowView.new(buf(p), first * stride, stride), c, K.RowView.new(buf(gates), first * 2 * width, 2 * width),
                    K.RowView.new(buf(gates), first * 2 * width + width, 2 * width))
            call = K.ChainBatch(weights, *rows, buf(conv), buf(st), K.StateOut.InPlace, K.RowView.new(buf(out), first * width, width))
            (call.launch_bf16_state if state == "bf16" else call.launch)(meta, K.Stream())
            torch.cuda.synchronize()
        return out, st

    got = run(K.Weights(h, buf(off(cw)), buf(a_log), buf(off(dtb)), buf(nw), 1e-5, -5.0), [list(range(n))])
    want = run(K.Weights(h, buf(cw), buf(a_log), buf(dtb), buf(nw), 1e-5, -5.0), [[i] for i in range(n) if lens[i]])
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
