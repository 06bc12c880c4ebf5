"""Rows, conv windows and states at any element, in launches of several units a block and on the small-block kernels: the bits of the
same values at aligned addresses.  (Aligned rows go by bulk copies, a block's first row's issued by the prologue's warps; aligned states in
vectors.)"""
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


def moved(t, per, shift):
    """The values of `t`, rows of `per`, a buffer further on by `shift` elements and with one element between rows if shift is odd."""
    pitch = per + shift % 2
    out = torch.zeros(shift + (t.numel() // per) * pitch + 8, dtype=t.dtype, device="cuda")
    out[shift:shift + (t.numel() // per) * pitch].view(-1, pitch)[:, :per] = t.view(-1, per)
    return out, pitch


def bits(t):
    return t.view(torch.int16)


@pytest.mark.parametrize("state", ["f32", "bf16"])
@pytest.mark.parametrize("lens", [[1] * 9, [2, 1, 0, 3, 1, 7, 1, 1]])
@pytest.mark.parametrize("rows_at, conv_at, state_at", [(1, 0, 0), (0, 1, 0), (3, 5, 1), (8, 8, 2), (2, 3, 3)])
def test_layer_calls(K, lens, rows_at, conv_at, state_at, state):
    h, g = 32, torch.Generator(device="cuda").manual_seed(sum(lens))
    c, width, total, n, per = K.channels(h), h * DK, sum(lens), len(lens), K.state_len(h)
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=g) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
    w = K.Weights(h, buf(rn(c * 4, 0.5)), buf(rn(h, 0.5, torch.float32)), buf(rn(width, 1.0, torch.float32)), buf(1 + rn(DK, 0.1)), 1e-5, -5.0)
    p, a, gate, conv = rn(total * (c + 64)), rn(total * width), rn(total * width), rn(n * 3 * c)
    states = rn(n * per, 0.3, torch.bfloat16 if state == "bf16" else torch.float32)

    def run(rows_at, conv_at, state_at):
        (pp, ps), (aa, as_), (gg, gs), (cc, cs), (ss, st) = (moved(t, m, x) for t, m, x in (
            (p, c + 64, rows_at), (a, width, rows_at), (gate, width, rows_at), (conv, 3 * c, conv_at), (states, per, state_at)))
        out = torch.full((total * width,), -1.0, dtype=torch.bfloat16, device="cuda")
        meta = K.BatchMeta.new(n)
        meta.set([K.Request(r, conv_at + i * cs, state_at + i * st) for i, r in enumerate(lens)])
        call = K.ChainBatch(w, K.RowView.new(buf(pp), rows_at, ps), c, K.RowView.new(buf(aa), rows_at, as_), K.RowView.new(buf(gg), rows_at, gs),
                            buf(cc), buf(ss), K.StateOut.InPlace, K.RowView.dense(buf(out), width))
        (call.launch_bf16_state if state == "bf16" else call.launch)(meta, K.Stream())
        torch.cuda.synchronize()
        return out, ss[state_at:state_at + n * st].view(n, st)[:, :per].contiguous()

    for x, y in zip(run(rows_at, conv_at, state_at), run(0, 0, 0)):
        assert torch.equal(bits(x), bits(y))


@pytest.mark.parametrize("state", ["f32", "bf16"])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_core_verify_and_replay(K, shift, state):
    core = importlib.import_module("glm53f-afd_b200.core")
    h, lens, keep, per = 5, [3, 1, 4], [2, 1, 0], 5 * DK * DK
    g, total = torch.Generator(device="cuda").manual_seed(shift), sum(lens)
    rn = lambda m: torch.randn(m, device="cuda", generator=g)
    n = total * h
    q, k = (torch.nn.functional.normalize(rn(n * DK).view(n, DK)).bfloat16().view(-1) for _ in range(2))
    v, glog, beta = rn(n * DK).bfloat16(), torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n))
    states = (rn(len(lens) * per) * 0.1).to(torch.bfloat16 if state == "bf16" else torch.float32)
    cu, kept = torch.tensor([0, 3, 4, 8], dtype=torch.int32, device="cuda"), torch.tensor(keep, dtype=torch.int32, device="cuda")

    def run(shift):
        ss, pitch = moved(states, per, shift)
        off = shift + torch.arange(len(lens), dtype=torch.int64, device="cuda") * pitch
        after, committed, out = ss.clone(), ss.clone(), torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda")
        saves = (torch.zeros(n * DK, device="cuda"), torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda"), torch.zeros(n * DK, device="cuda"),
                 torch.zeros(n, device="cuda"))
        core.decode_batch(h, total, cu, q, k, v, glog, beta, ss, off, state_out=after, out=out, saves=saves)
        core.commit_batch(h, 1, cu, kept, committed, 0, off, saves, n * DK, n)
        torch.cuda.synchronize()
        cut = lambda t: t[shift:shift + len(lens) * pitch].view(-1, pitch)[:, :per].contiguous()
        assert torch.equal(ss[:shift], after[:shift])
        return out, cut(after), cut(committed)

    for x, y in zip(run(shift), run(0)):
        assert torch.equal(bits(x), bits(y))


@pytest.mark.parametrize("state", ["f32", "bf16"])
@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("heads", [16, 64])  # one prompt's instance and that of many units
def test_exact_prefill(K, heads, shift, state):
    lens, g = [9, 21], torch.Generator(device="cuda").manual_seed(shift)
    c, width, total, n, per = K.channels(heads), heads * DK, sum(lens), len(lens), K.state_len(heads)
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=g) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
    w = K.Weights(heads, buf(rn(c * 4, 0.5)), buf(rn(heads, 0.5, torch.float32)), buf(rn(width, 1.0, torch.float32)), buf(1 + rn(DK, 0.1)), 1e-5, -5.0)
    p, gates, conv = rn(total * (c + 64)), rn(total * 2 * width), rn(n * 3 * c)
    states = rn(n * per, 0.3, torch.bfloat16 if state == "bf16" else torch.float32)
    K.set_prefill_form(K.Form.EXACT)

    def run(shift):
        ss, pitch = moved(states, per, shift)
        out = torch.full((total * width,), -1.0, dtype=torch.bfloat16, device="cuda")
        meta = K.BatchMeta.new(n)
        meta.set([K.Request(r, i * 3 * c, shift + i * pitch) for i, r in enumerate(lens)])
        call = K.PrefillBatch(w, K.RowView.dense(buf(p), c + 64), c, K.RowView.new(buf(gates), 0, 2 * width), K.RowView.new(buf(gates), width, 2 * width),
                              buf(conv.clone()), buf(ss), K.StateOut.InPlace, K.RowView.dense(buf(out), width), 0, K.PrefillWorkspace.new(heads, n, 16))
        (call.launch_bf16_state if state == "bf16" else call.launch)(meta, K.Stream())
        torch.cuda.synchronize()
        return out, ss[shift:shift + n * pitch].view(n, pitch)[:, :per].contiguous()

    for x, y in zip(run(shift), run(0)):
        assert torch.equal(bits(x), bits(y))
