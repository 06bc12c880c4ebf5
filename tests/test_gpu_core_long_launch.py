"""Core decode launches either side of the length from which a state's slot is given back late (csrc/kda_chain.cu, late_release):
a step of many slots leaves the bits of the same step made in small launches."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("state,slots", [("bf16", 31), ("bf16", 32), ("bf16", 40), ("bf16", 45), ("bf16", 46), ("f32", 15), ("f32", 16), ("f32", 21)])
def test_many_slots_have_the_bits_of_few(state, slots):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    core = importlib.import_module("glm53f-afd_b200.core")
    h, per = 64, 64 * DK * DK
    gen = torch.Generator(device="cuda").manual_seed(slots)
    rn = lambda n: torch.randn(n, device="cuda", generator=gen)
    n = slots * h
    q, k = (torch.nn.functional.normalize(rn(n * DK).view(n, DK)).bfloat16().view(-1) for _ in range(2))
    v, g, beta = rn(n * DK).bfloat16(), torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n))
    states = (rn(slots * per) * 0.1).to(torch.bfloat16 if state == "bf16" else torch.float32)

    def run(cuts):
        st, out = states.clone(), torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda")
        for a, b in zip(cuts, cuts[1:]):
            r, e = slice(a * h * DK, b * h * DK), slice(a * h, b * h)
            core.decode_batch(h, b - a, torch.arange(b - a + 1, dtype=torch.int32, device="cuda"), q[r], k[r], v[r], g[r], beta[e], st,
                              torch.arange(a, b, dtype=torch.int64, device="cuda") * per, out=out[r])
        torch.cuda.synchronize()
        return st, out

    got, want = run([0, slots]), run(list(range(0, slots, 3)) + [slots])
    assert all(torch.equal(a.view(torch.int16), b.view(torch.int16)) for a, b in zip(got, want))


@pytest.mark.parametrize("state,early,late", [("bf16", (16, 40, 45), 46), ("f32", (5, 15), 16)])
def test_where_the_line_lies(state, early, late):
    """A line for each state type: 19.5 bf16 units a block and 6.75 f32 ones (slots of 64 heads on 148 SMs)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("slots counted for 148 SMs")
    from captured import launches

    core = importlib.import_module("glm53f-afd_b200.core")
    h, per = 64, 64 * DK * DK
    z = lambda m, d=torch.bfloat16: torch.zeros(m, dtype=d, device="cuda")
    states = z(late * per, torch.bfloat16 if state == "bf16" else torch.float32)
    q, g, beta, out, off = z(late * h * DK), z(late * h * DK, torch.float32), z(late * h, torch.float32), z(late * h * DK), torch.arange(late, dtype=torch.int64, device="cuda") * per

    def instance(slots):
        cu = torch.arange(slots + 1, dtype=torch.int32, device="cuda")
        step = lambda: core.decode_batch(h, slots, cu, q, q, q, g, beta, states, off[:slots], out=out)
        step()
        names, _ = launches(step)
        assert len(names) == 1 and "recurrent_kernel" in names[0], names
        return names[0]

    assert len({instance(n) for n in early}) == 1 and instance(late) != instance(early[0])
