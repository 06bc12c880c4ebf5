"""A workspace that holds the whole call is used in parts all the same; the results are those of a small one, walked in many parts."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("state, fused", [(torch.float32, True), (torch.bfloat16, False)])
@pytest.mark.parametrize("lens", [[4032, 70], [4033, 1], [8127, 4100], [8129, 0]])  # 63, 64, 127 and 128 chunks: one, two, two, three parts
def test_same_bits(lens, state, fused):
    core = importlib.import_module("glm53f-afd_b200.core")
    gen = torch.Generator(device="cuda").manual_seed(lens[0])
    heads, rows, per = 17, sum(lens), 17 * DK * DK
    n = rows * heads
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    q, k, v, beta = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16(), torch.sigmoid(rn(n))
    g, start = torch.nn.functional.logsigmoid(rn(n * DK) + 3), (rn(2 * per) * 0.05).to(state)
    cu, off = torch.tensor([0] + lens, device="cuda").cumsum(0).int(), torch.arange(2, device="cuda") * per
    extra = {"gate": rn(n * DK).bfloat16(), "norm_w": rn(DK).bfloat16(), "eps": 1e-5} if fused else {}

    def run(chunks):
        out, st = torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda"), start.clone()
        ws = torch.full((core.prefill_workspace_bytes(heads, 2, chunks),), 0xff, dtype=torch.uint8, device="cuda")
        core.prefill_varlen(heads, rows, cu, max(lens), q, k, v, g, beta, st, off, out=out, workspace=ws, **extra)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return out, st

    for a, b in zip(run(300), run(10)):
        assert torch.isfinite(a).all() and torch.equal(a, b)
