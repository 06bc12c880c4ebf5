"""Single-pass chunked prefill under output gates so low that their sigmoid is below the smallest normal f32: the outputs, which bf16 holds, are formed
from it and not lost."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("gate_value", [-80.0, -87.5, -88.5])
def test_faint_gates(gate_value):
    core = importlib.import_module("glm53f-afd_b200.core")
    heads, rows, eps = 2, 100, 1e-5
    gen = torch.Generator(device="cuda").manual_seed(8)
    n = rows * heads
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    q, k, v, g, beta = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16(), torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n))
    norm_w = torch.full((DK,), 4.0, dtype=torch.bfloat16, device="cuda")

    def run(**gated):
        out = torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda")
        core.prefill_varlen(heads, rows, torch.tensor([0, rows], dtype=torch.int32, device="cuda"), rows, q, k, v, g, beta,
                            torch.zeros(heads * DK * DK, device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda"), out=out, **gated)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return out.double().view(n, DK)

    y = run()  # the norm's input, in the bf16 that it is formed from
    gate = torch.full((n * DK,), gate_value, dtype=torch.bfloat16, device="cuda")
    want = 4.0 * y * (y.square().mean(1, keepdim=True) + eps).rsqrt() * torch.sigmoid(gate.double().view(n, DK))
    got = run(gate=gate, norm_w=norm_w, eps=eps)
    # bf16 of the result: half an ulp, at most 2^-8 of it (seven bits behind the leading one), or 2^-134 below the smallest normal; the exponential's own error is 2^-17 at these arguments
    assert bool(((got - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -15) + 2.0 ** -134).all())
    assert bool((got != 0).any())
