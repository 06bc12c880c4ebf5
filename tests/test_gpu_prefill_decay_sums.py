"""Chunked prefill under strong decays: a row's way into the final state is the exponential of the sum of the decays behind the row, and no longer sum's rounding.

One chunk whose rows have a key channel each, from a zero state: nothing of a row reaches another, beta is one and the keys are ones, so that every factor but
the decay is exact, and channel 2 i of the state is v_i exp(g_{i+1} + ... + g_63)."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK, ROWS = 128, 64


@pytest.mark.parametrize("heads, chunks", [(4, 0), (4, 8), (40, 8), (160, 8)])  # a block a chain; over a workspace: U in the items, in the walk, all in one launch
@pytest.mark.parametrize("decay", [0.7, 2.0, 4.0, 5.8])
def test_last_rows(decay, heads, chunks):
    core = importlib.import_module("glm53f-afd_b200.core")
    gen = torch.Generator(device="cuda").manual_seed(3)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    n = ROWS * heads
    k = torch.zeros(ROWS, heads, DK, device="cuda")
    k[torch.arange(ROWS), :, 2 * torch.arange(ROWS)] = 1.0
    q, v = rn(n * DK).mul(DK ** -0.5).bfloat16(), rn(ROWS, heads, DK).bfloat16()
    g = -decay * torch.exp(0.2 * rn(ROWS, heads, DK))
    cu, off = torch.tensor([0, ROWS], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda")
    state, out = torch.zeros(heads * DK * DK, device="cuda"), torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda")
    ws = torch.empty(core.prefill_workspace_bytes(heads, 1, chunks), dtype=torch.uint8, device="cuda") if chunks else None
    # a longer longest sequence than there is: short calls with a workspace run without it
    core.prefill_varlen(heads, ROWS, cu, 64 * 64 if chunks else ROWS, q, k.bfloat16().view(-1), v.view(-1), g.view(-1), torch.ones(n, device="cuda"), state, off,
                        out=out, workspace=ws)
    torch.cuda.synchronize()
    assert core.device_status() == 0
    after = g.double().flip(0).cumsum(0).flip(0) - g.double()  # the decays behind each row
    want = torch.zeros(heads, DK, DK, dtype=torch.float64, device="cuda")  # [head][value][key]
    for i in range(ROWS):
        want[:, :, 2 * i] = v[i].double() * after[i, :, 2 * i].exp()[:, None]
    # Two bf16 terms hold the row's factor to 2^-18; its exponentials, reciprocal and products, and the rounding of sums of a few decays (beyond the eighth row from
    # the end, the rows are too faint to count at e^-2 and more; at e^-0.7 the sums are small), 2^-20.
    assert (state.view(heads, DK, DK).double() - want).norm() <= (2.0 ** -18 + 2.0 ** -20) * want.norm()
