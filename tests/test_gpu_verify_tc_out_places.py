"""The chunked core verify with its output buffer at any element: the bits of the outputs on 16 bytes, which leave in vectors, and nothing written
beside them; one unit a block and several, with and without replay saves."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK, HEADS = 128, 64


@pytest.mark.parametrize("saved", [False, True])
@pytest.mark.parametrize("lens", [[3], [16, 1, 5, 16, 9, 2, 0, 12]])
def test_outputs(lens, saved):
    core = importlib.import_module("glm53f-afd_b200.core")
    gen = torch.Generator(device="cuda").manual_seed(len(lens))
    total, per, b = sum(lens), HEADS * DK * DK, len(lens)
    n = total * HEADS
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    rows = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16(), torch.nn.functional.logsigmoid(rn(n * DK) + 1), torch.sigmoid(rn(n))
    states, off = (rn(b * per) * 0.05).bfloat16(), torch.arange(b, device="cuda") * per
    cu = torch.tensor([0] + lens, device="cuda").cumsum(0).int()

    def run(at):
        buf = torch.full((at + n * DK + 16,), -1.0, dtype=torch.bfloat16, device="cuda")
        saves = (torch.zeros(n * DK, device="cuda"), torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda"), torch.zeros(n * DK, device="cuda"), torch.zeros(n, device="cuda"))
        core.decode_batch(HEADS, total, cu, *rows, states, off, state_out=None, flags=core.TENSOR, out=buf[at:], saves=saves if saved else None)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        assert bool((buf[:at] == -1).all()) and bool((buf[at + n * DK:] == -1).all())
        return [buf[at:at + n * DK].clone().view(torch.int16), saves[1].view(torch.int16), saves[0], saves[2], saves[3]]

    want = run(0)
    for at in (1, 2, 4, 7, 8, 9):
        assert all(torch.equal(x, y) for x, y in zip(run(at), want)), at
