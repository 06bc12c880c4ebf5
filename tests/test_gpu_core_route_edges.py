"""Core decode at the borders of the range of units that runs on two small blocks a unit (more than one and at most two units an SM): the bits of
each request alone, which runs on one."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("per_sm, more", [(1, 0), (1, 1), (2, 0), (2, 1)])
@pytest.mark.parametrize("heads", [1, 37])
def test_borders(heads, per_sm, more, bf16):
    core = importlib.import_module("glm53f-afd_b200.core")
    units = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    batch = (units + heads - 1) // heads if more else units // heads  # heads = 1 hits the border itself
    gen = torch.Generator(device="cuda").manual_seed(units)
    per, n = heads * DK * DK, batch * heads
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(batch, -1)
    rows = unit(DK ** -0.5), unit(1.0), rn(batch, heads * DK).bfloat16(), torch.nn.functional.logsigmoid(rn(batch, heads * DK) + 3), torch.sigmoid(rn(batch, heads))
    states = (rn(batch, per) * 0.05).to(torch.bfloat16 if bf16 else torch.float32)

    def run(a, b):
        st, out = states[a:b].clone(), torch.zeros(b - a, heads * DK, dtype=torch.bfloat16, device="cuda")
        core.decode_batch(heads, b - a, torch.arange(b - a + 1, device="cuda").int(), *(t[a:b].clone().view(-1) for t in rows), st.view(-1), torch.arange(b - a, device="cuda") * per,
                          out=out.view(-1))
        return out.view(torch.int16), st.view(torch.int16)

    out, st = run(0, batch)
    for i in range(batch):
        o, s = run(i, i + 1)
        assert torch.equal(o[0], out[i]) and torch.equal(s[0], st[i]), i
    torch.cuda.synchronize()
    assert core.device_status() == 0
