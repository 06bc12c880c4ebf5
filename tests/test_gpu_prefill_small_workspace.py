"""The chunked layer prefill with workspaces that hold fewer slots than there are chains: the requests go in two parts, with the
bits that a workspace of 64 rows gives; ragged batches, even and odd, with empty requests and windows that advance."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("state", ["f32", "bf16"])
@pytest.mark.parametrize("lens", [[70, 130, 7], [65, 0, 200], [1, 64, 100, 129, 0], [0, 0, 80]])
def test_two_parts_leave_the_bits_of_one(lens, state):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    K = importlib.import_module("glm53f-afd_b200.kernel")
    h, n, total = 2, len(lens), sum(lens)
    g = torch.Generator(device="cuda").manual_seed(total)
    c, width = K.channels(h), h * DK
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=g) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
    w = K.Weights(h, buf(rn(c * 4, 0.5)), buf(rn(h, 0.5, torch.float32)), buf(rn(width, 1.0, torch.float32)), buf(1 + rn(DK, 0.1)), 1e-5, -5.0)
    p, gates, conv = rn(total * (c + 8)), rn(total * 2 * width), rn(n * 3 * c)
    states = rn(n * K.state_len(h), 0.3, torch.bfloat16 if state == "bf16" else torch.float32)
    meta, got, before = K.BatchMeta.new(n), [], K.set_prefill_form(K.Form.CHUNKED)
    meta.set([K.Request(r, i * 3 * c, i * K.state_len(h)) for i, r in enumerate(lens)])
    try:
        for rows in (64, 48, 33, 32):  # 32: the exact form
            st, cv, out = states.clone(), conv.clone(), torch.full((total * width,), -1.0, dtype=torch.bfloat16, device="cuda")
            call = K.PrefillBatch(w, K.RowView.dense(buf(p), c + 8), c, K.RowView.new(buf(gates), 0, 2 * width), K.RowView.new(buf(gates), width, 2 * width),
                                  buf(cv), buf(st), K.StateOut.InPlace, K.RowView.dense(buf(out), width), 0, K.PrefillWorkspace.new(h, n, rows))
            (call.launch_bf16_state if state == "bf16" else call.launch)(meta, K.Stream())
            torch.cuda.synchronize()
            got.append((out, st, cv))
    finally:
        K.set_prefill_form(before)
    for other in got[1:3]:
        for a, b in zip(got[0], other):
            assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    assert not torch.equal(got[0][0].view(torch.int16), got[3][0].view(torch.int16)) and torch.equal(got[0][2].view(torch.int16), got[3][2].view(torch.int16))
