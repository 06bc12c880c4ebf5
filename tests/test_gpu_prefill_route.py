"""Which calls with a workspace run without it, one block a chain: those of few chunks, unless one long sequence among short ones would have too few blocks
at work.  A workspace of one byte's value is left as it was by the calls that do not use it."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("heads, lens, fused, alone", [
    (1, [192], False, True), (1, [193], False, False), (64, [192, 1], True, True),
    (64, [384, 1], True, True), (64, [385, 1], False, False), (14, [256] + [1] * 7, False, True), (14, [257] + [1] * 7, False, False), (112, [384], False, True),
    (64, [128, 1, 1, 1], False, True), (64, [129, 1, 1, 1], False, False), (64, [128, 1, 1, 1], True, False), (64, [64, 64, 64], False, False)])
def test_route(heads, lens, fused, alone):
    core = importlib.import_module("glm53f-afd_b200.core")
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines depend on the number of SMs")
    gen = torch.Generator(device="cuda").manual_seed(2)
    rows, n, per = sum(lens), sum(lens) * heads, heads * DK * DK
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    extra = {"gate": rn(n * DK).bfloat16(), "norm_w": rn(DK).bfloat16()} if fused else {}
    cu, off = torch.tensor([0] + lens, device="cuda").cumsum(0).int(), torch.arange(len(lens), device="cuda") * per
    ws = torch.full((core.prefill_workspace_bytes(heads, len(lens), 32),), 0x5a, dtype=torch.uint8, device="cuda")
    core.prefill_varlen(heads, rows, cu, max(lens), unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16(), -torch.rand(n * DK, device="cuda", generator=gen), torch.sigmoid(rn(n)),
                        torch.zeros(len(lens) * per, device="cuda"), off, out=torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda"), workspace=ws, **extra)
    torch.cuda.synchronize()
    assert core.device_status() == 0
    untouched = bool((ws == 0x5a).all())
    assert untouched == alone
