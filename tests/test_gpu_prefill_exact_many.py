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


@pytest.mark.parametrize("quarters, octet", [(3, False), (4, True)])
def test_which_kernel_takes_how_many_units(quarters, octet):
    """A unit is four blocks of rows_kernel: up to three of them on an SM a row's latency counts, beyond that the work of its warps."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from captured import launches

    K = importlib.import_module("glm53f-afd_b200.kernel")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    h, n = (quarters * sms // 4 - (0 if octet else 1)) // 2, 2
    c, width, total = K.channels(h), h * DK, 16 * n
    zb = lambda m: K.DeviceBuffer(torch.zeros(m, dtype=torch.bfloat16, device="cuda").view(torch.uint8))
    zf = lambda m: K.DeviceBuffer(torch.zeros(m, device="cuda").view(torch.uint8))
    w = K.Weights(h, zb(c * 4), zf(h), zf(width), zb(DK), 1e-5, -5.0)
    meta, gates, stride = K.BatchMeta.new(n), zb(total * 2 * width), (c + h + 7) // 8 * 8
    meta.set([K.Request(16, i * 3 * c, i * K.state_len(h)) for i in range(n)])
    call = K.PrefillBatch(w, K.RowView.dense(zb(total * stride), stride), c, K.RowView.new(gates, 0, 2 * width), K.RowView.new(gates, width, 2 * width),
                          zb(n * 3 * c), zf(n * K.state_len(h)), K.StateOut.InPlace, K.RowView.dense(zb(total * width), width), 0,
                          K.PrefillWorkspace.new(h, n, 16))
    call.launch(meta, K.Stream())
    names, _ = launches(lambda: call.launch(meta, K.Stream()))
    assert any("rows_octet_kernel" in x for x in names) == octet and any("rows_kernel" in x for x in names) != octet, names
