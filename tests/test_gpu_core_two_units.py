"""Core decode with more than one and at most two units an SM, which runs on small blocks: the bits of each request alone, which does not, at
the edges of that range, with windows of no to several rows, states at any element, in place, into another buffer and not written."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK, HEADS = 128, 16


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("state_at", [0, 3])
@pytest.mark.parametrize("lens", [[1] * 10, [1, 0, 2, 1, 5, 1, 1, 3, 0, 1], [1] * 18, [1] * 19])
@pytest.mark.parametrize("to", ["in place", "apart", "nowhere"])
def test_decode(lens, state_at, bf16, to):
    core = importlib.import_module("glm53f-afd_b200.core")
    gen = torch.Generator(device="cuda").manual_seed(len(lens))
    total, per = sum(lens), HEADS * DK * DK
    n = total * HEADS
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    rows = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16(), torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n))
    states = (rn(state_at + len(lens) * per) * 0.05).to(torch.bfloat16 if bf16 else torch.float32)

    def run(group):
        first, ls = sum(lens[:group[0]]), [lens[i] for i in group]
        st, other = states.clone(), torch.zeros_like(states)
        out = torch.zeros(max(sum(ls), 1) * HEADS * DK, dtype=torch.bfloat16, device="cuda")
        cut = [t[first * t.numel() // total:] for t in rows]
        core.decode_batch(HEADS, sum(ls), torch.tensor([0] + ls, device="cuda").cumsum(0).int(), *(t.clone() for t in cut), st,
                          torch.tensor([state_at + i * per for i in group], device="cuda"), state_out={"in place": "in_place", "apart": other, "nowhere": None}[to], out=out)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return out[:sum(ls) * HEADS * DK], [(other if to == "apart" else st)[state_at + i * per:state_at + (i + 1) * per] for i in group]

    out, st = run(list(range(len(lens))))
    alone = [run([i]) for i in range(len(lens)) if lens[i]]
    assert torch.equal(out.view(torch.int16), torch.cat([o for o, _ in alone]).view(torch.int16))
    for i, l in enumerate(lens):
        want = alone[sum(1 for x in lens[:i] if x)][1][0] if l else states[state_at + i * per:state_at + (i + 1) * per]
        assert torch.equal(st[i].view(torch.int16), want.contiguous().view(torch.int16)), i
