"""The exact layer prefill in passes over the workspace (prologue, recurrence on independent warps, output norm) against the
chain's single launch: the same bits in outputs, states and conv windows, at the edges of the passes and of the four-row
blocks of the prologue, for ragged batches with empty requests, in place and out of place."""
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
@pytest.mark.parametrize("lens, pass_rows", [([7], 16), ([8], 16), ([15, 16, 17], 16), ([33, 0, 48], 16), ([0, 64, 1, 100], 32), ([257], 256)])
@pytest.mark.parametrize("in_place", [True, False])
def test_passes_leave_the_chains_bits(K, lens, pass_rows, state, in_place):
    h, g = 3, torch.Generator(device="cuda").manual_seed(sum(lens) + pass_rows)
    c, width, total, n = K.channels(h), h * DK, sum(lens), len(lens)
    stride = c + 8
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=g) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
    w = K.Weights(h, buf(rn(c * 4, 0.5)), buf(rn(h, 0.5, torch.float32)), buf(rn(width, 1.0, torch.float32)), buf(1 + rn(DK, 0.1)), 1e-5, -5.0)
    p, gates, conv = rn(total * stride), rn(total * 2 * width), rn(n * 3 * c)
    states = rn(n * K.state_len(h), 0.3, torch.bfloat16 if state == "bf16" else torch.float32)
    meta = K.BatchMeta.new(n)
    meta.set([K.Request(r, i * 3 * c, i * K.state_len(h)) for i, r in enumerate(lens)])
    stream, got = K.Stream(), []
    for prefill in (True, False):
        st, cv, out, other = states.clone(), conv.clone(), torch.full((total * width,), -1.0, dtype=torch.bfloat16, device="cuda"), torch.zeros_like(states)
        so = K.StateOut.InPlace if in_place else K.StateOut.To(buf(other))
        rows = (K.RowView.dense(buf(p), stride), c, K.RowView.new(buf(gates), 0, 2 * width), K.RowView.new(buf(gates), width, 2 * width))
        view = K.RowView.dense(buf(out), width)
        if prefill:
            call = K.PrefillBatch(w, *rows, buf(cv), buf(st), so, view, 0, K.PrefillWorkspace.new(h, n, pass_rows))
        else:
            call = K.ChainBatch(w, *rows, buf(cv), buf(st), so, view)
        (call.launch_bf16_state if state == "bf16" else call.launch)(meta, stream)
        if not prefill:
            K.conv_shift_batch(h, 1, meta, buf(cv), 0, K.RowView.dense(buf(p), stride), 0, stream)
        torch.cuda.synchronize()
        got.append((out, st if in_place else other, cv))
    for a, b in zip(*got):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("back", [0, 1, 40])  # rows by which the outputs lie before the gate rows of the same buffer
def test_outputs_over_the_gate_rows(K, back):
    h, rows, g = 2, 70, torch.Generator(device="cuda").manual_seed(back)
    c, width = K.channels(h), h * DK
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=g) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
    w = K.Weights(h, buf(rn(c * 4, 0.5)), buf(rn(h, 0.5, torch.float32)), buf(rn(width, 1.0, torch.float32)), buf(1 + rn(DK, 0.1)), 1e-5, -5.0)
    p, a, gate, conv, state = rn(rows * (c + h * 4)), rn(rows * width), rn((back + rows) * width), rn(3 * c), rn(K.state_len(h), 0.3, torch.float32)
    meta, stream, got = K.BatchMeta.new(1), K.Stream(), []
    meta.set([K.Request(rows, 0, 0)])
    for over in (False, True):
        gates, st, cv = gate.clone(), state.clone(), conv.clone()
        out = gates if over else torch.zeros(rows * width, dtype=torch.bfloat16, device="cuda")
        K.PrefillBatch(w, K.RowView.dense(buf(p), c + h * 4), c, K.RowView.dense(buf(a), width), K.RowView.new(buf(gates), back * width, width), buf(cv), buf(st),
                       K.StateOut.InPlace, K.RowView.dense(buf(out), width), 0, K.PrefillWorkspace.new(h, 1, 32)).launch(meta, stream)
        torch.cuda.synchronize()
        got.append((out[:rows * width].clone(), st, cv))
    for x, y in zip(*got):
        assert torch.equal(x.view(torch.int16), y.view(torch.int16))
