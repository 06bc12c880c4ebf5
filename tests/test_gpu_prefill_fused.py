"""The fused prefill launch (every block takes chunks, then chains): more chains than SMs in the core entry point, and the chunked
layer prefill, at the edges of chunks, of the prologue's four-row warps and of passes, with empty sequences between."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.fixture(scope="module")
def core():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return importlib.import_module("glm53f-afd_b200.core")


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("lens", [[130, 0, 64, 200, 1], [63, 65, 320, 0]])
def test_core_sequences_do_not_depend_on_their_company(core, lens, bf16):
    heads, total, g = 64, sum(lens), torch.Generator(device="cuda").manual_seed(sum(lens))
    n, per = total * heads, heads * DK * DK
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    q, k, v = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16()
    lg, beta = torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n))
    states = (rn(len(lens) * per) * 0.05).to(torch.bfloat16 if bf16 else torch.float32)

    def run(group, chunks):  # the sequences of `group`, which follow one another
        st, first, ls = states.clone(), sum(lens[:group[0]]), [lens[i] for i in group]
        rows, at = sum(ls), lambda t, w: t[first * heads * w:(first + sum(ls)) * heads * w].clone()
        cu = torch.tensor([0] + ls, device="cuda").cumsum(0).int()
        off = torch.tensor([i * per for i in group], device="cuda")
        out = torch.zeros(rows * heads * DK, dtype=torch.bfloat16, device="cuda")
        ws = torch.full((core.prefill_workspace_bytes(heads, len(ls), chunks),), 0xff, dtype=torch.uint8, device="cuda")
        core.prefill_varlen(heads, rows, cu, max(ls), at(q, DK), at(k, DK), at(v, DK), at(lg, DK), at(beta, 1), st, off, out=out, workspace=ws)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return out, [st[i * per:(i + 1) * per] for i in group]

    alone = [run([i], 8) for i in range(len(lens)) if lens[i]]  # 64 chains: state and chunk roles on two halves
    want = torch.cat([o for o, _ in alone]), [s for _, ss in alone for s in ss]
    for chunks in (1, 2, 16):
        out, st = run(list(range(len(lens))), chunks)  # 256 chains or more: one launch a pass
        assert torch.equal(out.view(torch.int16), want[0].view(torch.int16)), chunks
        assert all(torch.equal(a, b) for a, b in zip([s for s, l in zip(st, lens) if l], want[1])), chunks


# Bounds as for the other chunked layer prefills: bf16 operands, 5e-2 of the largest output, 1e-2 and 1e-3 relative L2.
@pytest.mark.parametrize("lower", [-5.0, -0.05])
@pytest.mark.parametrize("lens, pass_rows", [([61, 0, 66], 64), ([67, 130, 3], 64), ([64, 255], 1024)])
def test_layer_prefill_agrees_with_the_exact_form(core, lens, pass_rows, lower):
    K = importlib.import_module("glm53f-afd_b200.kernel")
    h, g = 4, torch.Generator(device="cuda").manual_seed(sum(lens))
    c, width, total, n = K.channels(h), h * DK, sum(lens), len(lens)
    stride = c + 4
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=g) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
    w = K.Weights(h, buf(rn(c * 4, 0.5)), buf(rn(h, 0.5, torch.float32)), buf(rn(width, 1.0, torch.float32)), buf(1 + rn(DK, 0.1)), 1e-5, lower)
    p, gates, conv, states = rn(total * stride), rn(total * 2 * width), rn(n * 3 * c), rn(n * K.state_len(h), 0.3, torch.float32)
    meta = K.BatchMeta.new(n)
    meta.set([K.Request(r, i * 3 * c, i * K.state_len(h)) for i, r in enumerate(lens)])
    got = []
    for form in (K.Form.CHUNKED, K.Form.EXACT):
        st, cv, out = states.clone(), conv.clone(), torch.full((total * width + 64,), -1.0, dtype=torch.bfloat16, device="cuda")
        before = K.set_prefill_form(form)
        try:
            K.PrefillBatch(w, K.RowView.dense(buf(p), stride), c, K.RowView.new(buf(gates), 0, 2 * width), K.RowView.new(buf(gates), width, 2 * width),
                           buf(cv), buf(st), K.StateOut.InPlace, K.RowView.new(buf(out), 0, width), 0,
                           K.PrefillWorkspace.new(h, n, pass_rows)).launch(meta, K.Stream())
        finally:
            K.set_prefill_form(before)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        assert bool((out[total * width:] == -1).all())
        got.append((out[:total * width].float(), st, cv))
    (o1, s1, c1), (o2, s2, c2) = got
    assert not torch.equal(o1, o2)  # the chunked form did run
    assert (o1 - o2).abs().max() <= 5e-2 * o2.abs().max() and (o1 - o2).norm() <= 1e-2 * o2.norm()
    assert (s1 - s2).norm() <= 1e-3 * s2.norm() and torch.equal(c1, c2)
