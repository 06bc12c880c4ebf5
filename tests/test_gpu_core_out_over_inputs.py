"""Core decode and exact core verify whose outputs lie over the q, k or v rows: the bits of outputs elsewhere.  With more than one and at most two
units an SM, and with replay saves, other calls run on two blocks a unit."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK, HEADS = 128, 16


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("saved", [False, True])
@pytest.mark.parametrize("lens", [[1] * 10, [1] * 18, [2, 1, 7, 0, 3, 1, 16, 1, 1, 4], [5]])
def test_outputs_over_inputs(lens, saved, bf16):
    core = importlib.import_module("glm53f-afd_b200.core")
    gen = torch.Generator(device="cuda").manual_seed(len(lens))
    total, per = sum(lens), HEADS * DK * DK
    n = total * HEADS
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    rows = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16(), torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n))
    states = (rn(len(lens) * per) * 0.05).to(torch.bfloat16 if bf16 else torch.float32)
    cu, off = torch.tensor([0] + lens, device="cuda").cumsum(0).int(), torch.arange(len(lens), device="cuda") * per

    def run(over):
        st, t = states.clone(), [x.clone() for x in rows]
        out = torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda") if over is None else t[over]
        saves = (torch.zeros(n * DK, device="cuda"), torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda"), torch.zeros(n * DK, device="cuda"), torch.zeros(n, device="cuda"))
        core.decode_batch(HEADS, total, cu, *t, st, off, out=out, saves=saves if saved else None)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return [x.view(torch.int16) for x in (out, st, saves[1])] + [saves[0], saves[2], saves[3]]

    want = run(None)
    for over in (0, 1, 2):
        assert all(torch.equal(x, y) for x, y in zip(run(over), want)), "qkv"[over]
