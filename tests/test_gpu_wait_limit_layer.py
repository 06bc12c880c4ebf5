"""The same failure path in a layer call whose blocks meet windows of several rows and single rows: the warps of the prologue are
then in different units when a wait runs out, and all of them still leave.  Unit 0 never gets its state, so its rows stay in
the ring of cooked rows, and the first row that finds the ring full gives up (`glm53f_kda_debug_wait_test`, 1 ms)."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


# As many heads as SMs: block 0 has (0, head 0) and then a unit of the next request.  Rows beyond the ring
# (6 rows with f32 states, 10 with bf16) put the waits that run out into different warps; [2, 1, 9] ends among single rows; one request alone
# is a launch of one unit a block.  bf16 launches of several units a block have two teams of four warps, which take single rows in turn: in
# [13, 1, 1] and [15, 1, 1, 1] rows 12 to 14 of the window, stuck behind the ring, are those of warps 4 to 6, which then meet their
# own team's vote.
@pytest.mark.parametrize("state", ["f32", "bf16"])
@pytest.mark.parametrize("lens", [[6, 1], [9, 1, 1], [11, 1], [2, 1, 9], [8, 3, 1], [8], [9], [11], [12], [13, 1, 1], [15, 1, 1, 1]])
def test_every_warp_leaves_when_a_wait_runs_out(pkg, lens, state):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    K, core = (importlib.import_module("glm53f-afd_b200." + m) for m in ("kernel", "core"))
    lib = pkg.ffi.load()
    h, n, total = torch.cuda.get_device_properties(0).multi_processor_count, len(lens), sum(lens)
    g = torch.Generator(device="cuda").manual_seed(total)
    c, width, per = K.channels(h), h * DK, K.state_len(h)
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=g) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
    w = K.Weights(h, buf(rn(c * 4, 0.5)), buf(rn(h, 0.5, torch.float32)), buf(rn(width, 1.0, torch.float32)), buf(1 + rn(DK, 0.1)), 1e-5, -5.0)
    stride = c + h + 4
    p, gates, conv = rn(total * stride), rn(total * 2 * width), rn(n * 3 * c)
    states = rn(n * per, 0.3, torch.bfloat16 if state == "bf16" else torch.float32)
    meta, stream = K.BatchMeta.new(n), K.Stream()
    meta.set([K.Request(r, i * 3 * c, i * per) for i, r in enumerate(lens)])

    def launch():
        st, out = states.clone(), torch.zeros(total * width, dtype=torch.bfloat16, device="cuda")
        call = K.ChainBatch(w, K.RowView.dense(buf(p), stride), c, K.RowView.new(buf(gates), 0, 2 * width), K.RowView.new(buf(gates), width, 2 * width),
                            buf(conv), buf(st), K.StateOut.InPlace, K.RowView.dense(buf(out), width))
        (call.launch_bf16_state if state == "bf16" else call.launch)(meta, stream)
        torch.cuda.synchronize()
        return out.view(total, h, DK).view(torch.int16), st.view(n, h, -1)

    clean_out, clean_st = launch()
    assert core.device_status() == 0
    assert lib.glm53f_kda_debug_wait_test(1_000_000, 1) == 0
    try:
        out, st = launch()
        assert 101 <= core.device_status() <= 108 and core.device_status() == 0
        # block 0 has head 0 of every request; the other heads are a clean launch's
        assert torch.equal(out[:, 1:], clean_out[:, 1:]) and torch.equal(st[:, 1:], clean_st[:, 1:])
        assert torch.equal(st[:, 0], states.view(n, h, -1)[:, 0])
        again = launch()
        assert core.device_status() == 0 and torch.equal(again[0], clean_out) and torch.equal(again[1], clean_st)
    finally:
        assert lib.glm53f_kda_debug_wait_test(0, 0) == 0
