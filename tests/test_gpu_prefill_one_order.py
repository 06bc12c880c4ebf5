"""The core prefill by one block a chain against the recurrence in 64 bits: short calls with a workspace, and blocks that take the longest sequences first, at
the most sequences that are put in order (32) and one more."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("state", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads, lens, chunks", [
    (3, [192, 1, 65], 8), (40, [128, 2, 100, 64], 8), (75, [384, 70], 8),
    (5, [7 * i % 150 for i in range(32)], 0), (5, [7 * i % 150 for i in range(33)], 0), (149, [130], 0)])
def test_against_64_bits(heads, lens, chunks, state):
    core = importlib.import_module("glm53f-afd_b200.core")
    gen = torch.Generator(device="cuda").manual_seed(len(lens))
    total, per, batch = sum(lens), heads * DK * DK, len(lens)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(total, heads, DK), dim=2).mul(s).bfloat16()
    q, k, v, beta = unit(DK ** -0.5), unit(1.0), rn(total, heads, DK).bfloat16(), torch.sigmoid(rn(total, heads))
    g = torch.nn.functional.logsigmoid(rn(total, heads, DK) + 3)
    start = (rn(batch, heads, DK, DK) * 0.05).to(state)
    out, st = torch.zeros(total * heads * DK, dtype=torch.bfloat16, device="cuda"), start.clone()
    ws = torch.empty(core.prefill_workspace_bytes(heads, batch, chunks), dtype=torch.uint8, device="cuda") if chunks else None
    cu, off = torch.tensor([0] + lens, device="cuda").cumsum(0).int(), torch.arange(batch, device="cuda") * per
    core.prefill_varlen(heads, total, cu, max(lens), *(x.view(-1) for x in (q, k, v, g, beta)), st.view(-1), off, out=out, workspace=ws)
    torch.cuda.synchronize()
    assert core.device_status() == 0
    got, q, k, v, e, beta, s = out.view(total, heads, DK).double(), q.double(), k.double(), v.double(), g.double().exp(), beta.double(), start.double()
    # all sequences a row at a time; those that have ended keep their states
    first, length, want = cu[:-1].long(), torch.tensor(lens, device="cuda"), torch.zeros(total, heads, DK, dtype=torch.float64, device="cuda")
    for t in range(max(lens)):
        b = (length > t).nonzero()[:, 0]
        r = first[b] + t
        x = s[b] * e[r][:, :, None, :]
        x = x + (beta[r][:, :, None] * (v[r] - (x * k[r][:, :, None, :]).sum(-1)))[..., None] * k[r][:, :, None, :]
        s[b], want[r] = x, (x * q[r][:, :, None, :]).sum(-1)
    # The chunked form's bounds: outputs an ulp of bf16 of the largest and 5e-3 of the norm, FP32 states 1e-3; a bf16 state is rounded once a chunk, 2^-9 each
    assert float((got - want).abs().max() / want.abs().max()) <= 1 / 128
    rel = float((got - want).norm() / want.norm())
    assert rel <= 5e-3 if state is torch.float32 else rel <= 1e-2
    assert float((st.double() - s).norm() / s.norm()) <= (1e-3 if state is torch.float32 else 7 * 2.0 ** -9)
