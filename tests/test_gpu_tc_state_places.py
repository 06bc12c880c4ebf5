"""The chunked verify and commit with states at a multiple of a row (which come and go in boxes), on 16 bytes, and at any element, side by side in
one launch and several units a block: the bits of the same states at multiples of a row."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK, HEADS = 128, 64


@pytest.mark.parametrize("apart", [False, True])
@pytest.mark.parametrize("base", [0, 8, 1])
@pytest.mark.parametrize("lens", [[3], [16, 1, 5, 16, 9, 2, 0, 12]])
def test_states(lens, base, apart):
    core = importlib.import_module("glm53f-afd_b200.core")
    K = importlib.import_module("glm53f-afd_b200.kernel")
    gen = torch.Generator(device="cuda").manual_seed(len(lens))
    total, per, b = sum(lens), HEADS * DK * DK, len(lens)
    n = total * HEADS
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    rows = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16(), torch.nn.functional.logsigmoid(rn(n * DK) + 1), torch.sigmoid(rn(n))
    states = (rn(b, per) * 0.05).bfloat16()
    cu = torch.tensor([0] + lens, device="cuda").cumsum(0).int()
    keep = torch.tensor([max(0, m - i % 3) for i, m in enumerate(lens)], dtype=torch.int32, device="cuda")

    def run(gaps, base):  # gaps[i] elements in front of state i
        at, offs = 0, []
        for g in gaps:
            offs.append(at + g)
            at += g + per
        buf = torch.zeros(base + at + 8, dtype=torch.bfloat16, device="cuda")[base:]
        for o, s in zip(offs, states):
            buf[o:o + per] = s
        off = torch.tensor(offs, device="cuda")
        out = torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda")
        saves = (torch.zeros(n * DK, device="cuda"), torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda"), torch.zeros(n * DK, device="cuda"), torch.zeros(n, device="cuda"))
        core.decode_batch(HEADS, total, cu, *rows, buf, off, state_out=None, flags=core.TENSOR, out=out, saves=saves)
        to = torch.full_like(buf, -1.0) if apart else buf
        before = K.set_commit_form(K.Form.CHUNKED)
        try:
            core.commit_batch(HEADS, 1, cu, keep, buf, buf.numel(), off, saves, n * DK, n, state_out=to)
        finally:
            K.set_commit_form(before)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        got = torch.stack([to[o:o + per] for o in offs])
        rest = torch.ones(to.numel(), dtype=torch.bool, device="cuda")
        for o in offs:
            rest[o:o + per] = False
        assert bool((to[rest] == (-1.0 if apart else 0.0)).all())  # nothing beside the states was written
        return [t.view(torch.int16) for t in (out, got, saves[1])] + [saves[0], saves[2], saves[3]]

    want = run([0] * b, 0)
    for gaps in ([128] * b, [8] * b, [3] * b, [(0, 5, 128, 16, 8, 256, 1, 0)[i % 8] for i in range(b)]):
        assert all(torch.equal(x, y) for x, y in zip(run(gaps, base), want)), gaps
