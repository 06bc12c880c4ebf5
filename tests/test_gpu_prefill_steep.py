"""Chunked prefill where the decay of a block of sixteen rows is past the smallest normal number but two neighbouring rows across the
blocks' border decay by nothing: the pair's factor e^0 is formed as e^+46 x e^-93 x e^+47, of which none may vanish."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("workspace", [False, True])
@pytest.mark.parametrize("decay", [-5.8, -6.2])
def test_steep_blocks(decay, workspace):
    core = importlib.import_module("glm53f-afd_b200.core")
    heads, rows, gen = 2, 128, torch.Generator().manual_seed(5)
    rn = lambda *s: torch.randn(*s, generator=gen, dtype=torch.float64)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q, k, v, beta = unit(rn(rows, heads, DK)) * DK ** -0.5, unit(rn(rows, heads, DK)), rn(rows, heads, DK), torch.full((rows, heads), 0.9, dtype=torch.float64)
    k[16::16], q[16::16] = k[15:-1:16], k[15:-1:16]  # the first row of a block is the last of the one before again
    g = torch.full((rows, heads, DK), decay, dtype=torch.float64)
    g[16::16] = -0.01
    q, k, v = q.bfloat16().double(), k.bfloat16().double(), v.bfloat16().double()
    s, want = torch.zeros(heads, DK, DK, dtype=torch.float64), []
    for t in range(rows):  # state [head][value][key]
        s = s * g[t].float().double().exp()[:, None, :]
        s = s + (beta[t][:, None] * (v[t] - (s * k[t][:, None, :]).sum(-1)))[:, :, None] * k[t][:, None, :]
        want.append((s * q[t][:, None, :]).sum(-1))
    want = torch.stack(want)
    dev = lambda x, d: x.to(d).contiguous().cuda().view(-1)
    out, state = torch.zeros(rows * heads * DK, dtype=torch.bfloat16, device="cuda"), torch.zeros(heads * DK * DK, device="cuda")
    ws = torch.empty(core.prefill_workspace_bytes(heads, 1, 2), dtype=torch.uint8, device="cuda") if workspace else None
    core.prefill_varlen(heads, rows, torch.tensor([0, rows], dtype=torch.int32, device="cuda"), rows, dev(q, torch.bfloat16), dev(k, torch.bfloat16), dev(v, torch.bfloat16),
                        dev(g, torch.float32), dev(beta, torch.float32), state, torch.zeros(1, dtype=torch.int64, device="cuda"), out=out, workspace=ws)
    torch.cuda.synchronize()
    assert core.device_status() == 0
    got = out.view(rows, heads, DK).double().cpu()
    # bf16 operands: the bound of the other chunked prefill tests, 1e-2 of the norm; a lost pair is 0.9 of its row
    assert (got - want).norm() <= 1e-2 * want.norm()
    assert (state.view(heads, DK, DK).double().cpu() - s).norm() <= 2e-3 * s.norm()


@pytest.mark.parametrize("decay, status", [(-12.0, 0), (-13.0, 121)])
@pytest.mark.parametrize("kind", ["single pass", "workspace", "verify"])
def test_decay_behind_a_middle_row(kind, decay, status):
    """Seven rows behind a block's middle row: e^-84 can be split into factors, e^-91 cannot and is reported."""
    core = importlib.import_module("glm53f-afd_b200.core")
    heads, rows, gen = 2, 16 if kind == "verify" else 70, torch.Generator(device="cuda").manual_seed(6)
    n = rows * heads * DK
    rn = lambda m, s=1.0: (torch.randn(m, device="cuda", generator=gen) * s)
    q, k, v, beta = rn(n, 0.01).bfloat16(), rn(n, 0.08).bfloat16(), rn(n).bfloat16(), torch.sigmoid(rn(rows * heads))
    g = torch.full((rows, heads * DK), -0.1, device="cuda")
    g[9:16] = decay
    cu, off, out = torch.tensor([0, rows], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros(n, dtype=torch.bfloat16, device="cuda")
    if kind == "verify":
        core.decode_batch(heads, rows, cu, q, k, v, g.view(-1), beta, rn(heads * DK * DK, 0.05).bfloat16(), off, state_out=None, flags=core.TENSOR, out=out)
    else:
        ws = torch.empty(core.prefill_workspace_bytes(heads, 1, 2), dtype=torch.uint8, device="cuda") if kind == "workspace" else None
        core.prefill_varlen(heads, rows, cu, rows, q, k, v, g.view(-1), beta, torch.zeros(heads * DK * DK, device="cuda"), off, out=out, workspace=ws)
    torch.cuda.synchronize()
    assert core.device_status() == status
    assert core.device_status() == 0
    assert bool(torch.isfinite(out).all())
