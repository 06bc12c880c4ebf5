"""Chunked prefill over a workspace under output gates so low that their sigmoid is below the smallest normal f32: the outputs, which bf16 holds, are not lost,
and are those of the call without a workspace, bit for bit."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("gate_value", [-80.0, -87.5, -88.5, None])  # None: all of a range around the border
@pytest.mark.parametrize("heads", [2, 40, 160])  # U in the items, in the walk, all in one launch
def test_faint_gates(heads, gate_value):
    core = importlib.import_module("glm53f-afd_b200.core")
    rows, eps = 100, 1e-5
    gen = torch.Generator(device="cuda").manual_seed(8)
    n = rows * heads
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    q, k, v, g, beta = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16(), torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n))
    norm_w = torch.full((DK,), 4.0, dtype=torch.bfloat16, device="cuda")
    gate = rn(n * DK).mul(3.0).sub(86.0).bfloat16() if gate_value is None else torch.full((n * DK,), gate_value, dtype=torch.bfloat16, device="cuda")

    def run(longest, chunks, **gated):
        out = torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda")
        ws = torch.empty(core.prefill_workspace_bytes(heads, 1, chunks), dtype=torch.uint8, device="cuda") if chunks else None
        core.prefill_varlen(heads, rows, torch.tensor([0, rows], dtype=torch.int32, device="cuda"), longest, q, k, v, g, beta,
                            torch.zeros(heads * DK * DK, device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda"), out=out, workspace=ws, **gated)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return out

    y = run(rows, 0).double().view(n, DK)  # the norm's input, in the bf16 that it is formed from
    want = 4.0 * y * (y.square().mean(1, keepdim=True) + eps).rsqrt() * torch.sigmoid(gate.double().view(n, DK))
    fused = {"gate": gate, "norm_w": norm_w, "eps": eps}
    got = run(64 * 64, 8, **fused)  # a longer longest sequence than there is: short calls with a workspace run without it
    # The bound of the call without a workspace: half an ulp of bf16, the exponential's own error, half of the smallest denormal; where the exponential overflows (below
    # -88.73) the sigmoid is zero
    lost = (gate.view(n, DK) < -88.7) & (got.view(n, DK) == 0)
    assert bool((((got.view(n, DK).double() - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -15) + 2.0 ** -134) | lost).all())
    assert bool((got != 0).any())
    assert torch.equal(got.view(torch.int16), run(rows, 0, **fused).view(torch.int16))
