"""The exact layer prefill of many units at once (rows_octet_kernel in csrc/kda_rows.cu) against the chain's single launch: the same
bits in outputs and states, at the edges of the groups of four rows that arrive together and of the passes, with empty requests."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("state", ["f32", "bf16"])
@pytest.mark.parametrize("lens, pass_rows", [([8, 9], 16), ([11, 1, 12], 16), ([0, 13, 4, 5], 32), ([33, 18], 16), ([70, 131], 64)])
@pytest.mark.parametrize("in_place", [True, False])
def test_many_units_have_the_chains_bits(lens, pass_rows, state, in_place):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    K = importlib.import_module("glm53f-afd_b200.kernel")
    h, g = 48, torch.Generator(device="cuda").manual_seed(sum(lens))
    c, width, total, n = K.channels(h), h * DK, sum(lens), len(lens)
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=g) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
    w = K.Weights(h, buf(rn(c * 4, 0.5)), buf(rn(h, 0.5, torch.float32)), buf(rn(width, 1.0, torch.float32)), buf(1 + rn(DK, 0.1)), 1e-5, -5.0)
    stride = c + 64
    p, gates, conv = rn(total * stride), rn(total * 2 * width), rn(n * 3 * c)
    states = rn(n * K.state_len(h), 0.3, torch.bfloat16 if state == "bf16" else torch.float32)
    meta = K.BatchMeta.new(n)
    meta.set([K.Request(r, i * 3 * c, i * K.state_len(h)) for i, r in enumerate(lens)])
    got = []
    for prefill in (True, False):
        st, other, out = states.clone(), torch.zeros_like(states), torch.full((total * width,), -1.0, dtype=torch.bfloat16, device="cuda")
        rows = (K.RowView.dense(buf(p), stride), c, K.RowView.new(buf(gates), 0, 2 * width), K.RowView.new(buf(gates), width, 2 * width))
        args = (w, *rows, buf(conv.clone()), buf(st), K.StateOut.InPlace if in_place else K.StateOut.To(buf(other)), K.RowView.dense(buf(out), width))
        call = K.PrefillBatch(*args, 0, K.PrefillWorkspace.new(h, n, pass_rows)) if prefill else K.ChainBatch(*args)
        (call.launch_bf16_state if state == "bf16" else call.launch)(meta, K.Stream())
        torch.cuda.synchronize()
        got.append((out, st if in_place else other))
    for a, b in zip(*got):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
