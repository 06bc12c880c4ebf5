"""The walk of several chains by one block: states at any element and into another buffer, gate rows on 16 bytes (which come by tensor copies)
and off them, empty and partial chunks between: the bits of each sequence alone."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK, HEADS = 128, 64


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("lens", [[64, 0, 129, 1], [0, 200, 0, 0, 64, 63, 128, 320]])
@pytest.mark.parametrize("state_at, gated", [(0, False), (0, True), (3, True), (8, False)])
def test_chains_of_a_block(lens, bf16, state_at, gated):
    core = importlib.import_module("glm53f-afd_b200.core")
    gen = torch.Generator(device="cuda").manual_seed(len(lens) + state_at)
    total, per = sum(lens), HEADS * DK * DK
    n = total * HEADS
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    q, k, v = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16()
    lg, beta, gate = torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n)), rn(n * DK).bfloat16()
    norm_w = (1 + 0.1 * rn(DK)).bfloat16() if gated else None
    states = (rn(len(lens) * per) * 0.05).to(torch.bfloat16 if bf16 else torch.float32)

    def run(group, chunks, at, apart):
        first, ls = sum(lens[:group[0]]), [lens[i] for i in group]
        cut = lambda t, w: t[first * HEADS * w:(first + sum(ls)) * HEADS * w].clone()
        st = torch.cat([torch.zeros(at, dtype=states.dtype, device="cuda"), states])
        to = torch.zeros_like(st) if apart else st
        cu, off = torch.tensor([0] + ls, device="cuda").cumsum(0).int(), torch.tensor([at + i * per for i in group], device="cuda")
        out = torch.zeros(sum(ls) * HEADS * DK, dtype=torch.bfloat16, device="cuda")
        ws = torch.full((core.prefill_workspace_bytes(HEADS, len(ls), chunks),), 0xff, dtype=torch.uint8, device="cuda")
        core.prefill_varlen(HEADS, sum(ls), cu, max(ls), cut(q, DK), cut(k, DK), cut(v, DK), cut(lg, DK), cut(beta, 1), st, off, state_out=to,
                            gate=cut(gate, DK) if gated else None, norm_w=norm_w, out=out, workspace=ws)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return out, [to[at + i * per:at + (i + 1) * per] for i in group]

    full = [i for i in range(len(lens)) if lens[i]]
    alone = [run([i], 8, 0, False) for i in full]
    for chunks in (1, 3, 8):
        out, st = run(list(range(len(lens))), chunks, state_at, True)
        assert torch.equal(out.view(torch.int16), torch.cat([o for o, _ in alone]).view(torch.int16)), chunks
        for i in range(len(lens)):
            want = alone[full.index(i)][1][0] if lens[i] else states[i * per:(i + 1) * per]
            assert torch.equal(st[i], want), (chunks, i)


@pytest.mark.parametrize("lens", [[64, 130, 256], [320, 1, 64, 127]])
@pytest.mark.parametrize("gate_at, gap", [(1, 0), (8, 8), (0, 1), (0, 4)])
def test_gate_rows_of_the_layer_form(lens, gate_at, gap):
    """The output gate's rows at any element and distance: the bits of rows on 16 bytes."""
    K = importlib.import_module("glm53f-afd_b200.kernel")
    core = importlib.import_module("glm53f-afd_b200.core")
    h, gen = HEADS, torch.Generator(device="cuda").manual_seed(sum(lens))
    c, width, total, n, per = K.channels(h), h * DK, sum(lens), len(lens), K.state_len(h)
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=gen) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
    w = K.Weights(h, buf(rn(c * 4, 0.5)), buf(rn(h, 0.5, torch.float32)), buf(rn(width, 1.0, torch.float32)), buf(1 + rn(DK, 0.1)), 1e-5, -5.0)
    p, a, gate, conv, state = rn(total * (c + h)), rn(total * width), rn(total * width), rn(n * 3 * c), rn(n * per, 0.05)
    K.set_prefill_form(K.Form.CHUNKED)

    def run(at, gap):
        rows = torch.zeros(at + total * (width + gap) + 8, dtype=torch.bfloat16, device="cuda")
        rows[at:at + total * (width + gap)].view(total, -1)[:, :width] = gate.view(total, -1)
        st, cv, out, meta, stream = state.clone(), conv.clone(), torch.zeros(total * width, dtype=torch.bfloat16, device="cuda"), K.BatchMeta.new(n), K.Stream()
        meta.set([K.Request(m, i * 3 * c, i * per) for i, m in enumerate(lens)])
        K.PrefillBatch(w, K.RowView.dense(buf(p), c + h), c, K.RowView.dense(buf(a), width), K.RowView.new(buf(rows), at, width + gap), buf(cv), buf(st),
                       K.StateOut.InPlace, K.RowView.dense(buf(out), width), 0, K.PrefillWorkspace.new(h, n, 256)).launch_bf16_state(meta, stream)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return out, st

    try:
        want = run(0, 0)
        assert all(torch.equal(x.view(torch.int16), y.view(torch.int16)) for x, y in zip(run(gate_at, gap), want))
    finally:
        K.set_prefill_form(K.Form.EXACT)


@pytest.mark.parametrize("lens", [[320, 320, 320], [700, 260, 301], [256, 300, 64, 500, 257]])
def test_blocks_that_leave_the_last_items_to_others(lens):
    """Chains that do not divide evenly by the SMs, four chunks and more each: the bits of each sequence alone, in every one of many launches."""
    core = importlib.import_module("glm53f-afd_b200.core")
    gen = torch.Generator(device="cuda").manual_seed(sum(lens))
    total, per = sum(lens), HEADS * DK * DK
    n = total * HEADS
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    rows = (unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16(), torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n)))

    def run(first, ls, launches):
        m, st = first * HEADS, torch.zeros(len(ls) * per, device="cuda")
        cut = [t[m * w:(m + sum(ls) * HEADS) * w].clone() for t, w in zip(rows, (DK, DK, DK, DK, 1))]
        cu, off = torch.tensor([0] + ls, device="cuda").cumsum(0).int(), torch.arange(len(ls), device="cuda") * per
        ws = torch.zeros(core.prefill_workspace_bytes(HEADS, len(ls), (max(ls) + 63) // 64), dtype=torch.uint8, device="cuda")
        outs = [torch.zeros(sum(ls) * HEADS * DK, dtype=torch.bfloat16, device="cuda") for _ in range(launches)]
        for out in outs:
            st.zero_()
            core.prefill_varlen(HEADS, sum(ls), cu, max(ls), *cut, st, off, out=out, workspace=ws)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return outs, st

    alone = [run(sum(lens[:i]), [ls], 1) for i, ls in enumerate(lens)]
    want, states = torch.cat([o[0] for o, _ in alone]).view(torch.int16), torch.cat([s for _, s in alone])
    outs, st = run(0, lens, 10)
    assert all(torch.equal(o.view(torch.int16), want) for o in outs) and torch.equal(st, states)
