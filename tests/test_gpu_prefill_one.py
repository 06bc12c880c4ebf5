"""The core prefill by one block a chain, with and without a workspace, against the two roles over a workspace: a call that gives a longer longest
sequence than there is takes those.  The same products and sums, so the same bits; rows behind a sequence's last are not numbers."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("gates", [3.0, -3.0])  # one reference row a chunk, one in sixteen
@pytest.mark.parametrize("state, fused", [(torch.float32, False), (torch.bfloat16, True)])
@pytest.mark.parametrize("heads, lens", [(1, [1]), (3, [63]), (3, [64, 65]), (2, [128, 1, 129]), (3, [0, 192, 64, 0]), (64, [2, 384]), (50, [300, 64, 7, 130]), (40, [70, 0, 64, 70, 129]), (57, [64, 192, 1, 130])])
def test_same_bits(heads, lens, state, fused, gates):
    core = importlib.import_module("glm53f-afd_b200.core")
    gen = torch.Generator(device="cuda").manual_seed(sum(lens))
    rows, per, batch = sum(lens), heads * DK * DK, len(lens)
    n = (rows + 64) * heads
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    q, k, v, beta = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16(), torch.sigmoid(rn(n))
    g, gate = torch.nn.functional.logsigmoid(rn(n * DK) + gates), rn(n * DK).bfloat16()
    for x in (q, k, v, g, gate):
        x[rows * heads * DK:] = float("nan")
    beta[rows * heads:] = float("nan")
    start = (rn(batch * per) * 0.05).to(state)
    cu, off = torch.tensor([0] + lens, device="cuda").cumsum(0).int(), torch.arange(batch, device="cuda").flip(0) * per
    extra = {"gate": gate, "norm_w": rn(DK).bfloat16(), "eps": 1e-5} if fused else {}

    def run(longest, chunks):
        out, st = torch.full((n * DK,), 7.0, dtype=torch.bfloat16, device="cuda"), start.clone()
        ws = torch.full((core.prefill_workspace_bytes(heads, batch, chunks),), 0xff, dtype=torch.uint8, device="cuda") if chunks else None
        core.prefill_varlen(heads, rows, cu, longest, q, k, v, g, beta, st, off, out=out, workspace=ws, **extra)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        assert bool((out[rows * heads * DK:] == 7.0).all())
        return out[:rows * heads * DK], st

    want = run(64 * 64, 8)
    for got in (run(max(lens), 8), run(max(lens), 0)):
        for a, b in zip(got, want):
            assert torch.isfinite(a).all() and torch.equal(a, b)
