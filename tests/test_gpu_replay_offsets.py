"""The commit replay whose saved values start at any element: all run on the small-block kernel (csrc/kda_chain.cu,
replay_entry), with the bits of aligned values.  Prefix lengths around the rows kept in flight."""
import ctypes
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("rows", [0, 1, 2, 3, 4, 5, 17])
@pytest.mark.parametrize("shift", [1, 2, 4])
def test_values_at_any_element(rows, shift):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ffi = importlib.import_module("glm53f-afd_b200.ffi")
    lib, h = ffi.load(), 6
    gen = torch.Generator(device="cuda").manual_seed(rows)
    n = max(rows, 1) * h
    k = torch.nn.functional.normalize(torch.randn(n, DK, device="cuda", generator=gen))
    v = torch.randn(n * DK, device="cuda", generator=gen).bfloat16()
    g = torch.exp(torch.nn.functional.logsigmoid(torch.randn(n * DK, device="cuda", generator=gen) + 3))
    beta = torch.sigmoid(torch.randn(n, device="cuda", generator=gen))
    state = torch.randn(h * DK * DK, device="cuda", generator=gen)
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def run(vv):
        out = torch.full_like(state, -1.0)
        assert lib.glm53f_kda_replay(h, rows, p(state), p(out), p(k), p(vv), p(g), p(beta), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        torch.cuda.synchronize()
        return out

    moved = torch.zeros(n * DK + 8, dtype=torch.bfloat16, device="cuda")
    moved[shift:shift + n * DK] = v
    got, want = run(moved[shift:]), run(v)
    assert torch.equal(got, want) and (rows > 0 or torch.equal(got, state))


@pytest.mark.parametrize("state", ["f32", "bf16"])
@pytest.mark.parametrize("shift", [0, 1, 2, 3, 4])
def test_a_batch_of_layers_on_the_small_block_kernel(shift, state):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from captured import launches

    core = importlib.import_module("glm53f-afd_b200.core")
    h, layers, keep = 3, 4, [4, 0, 7, 1]  # 48 units: more than find an SM for each of their blocks
    rows, n, per = [5, 2, 7, 3], 17 * h, h * DK * DK
    gen = torch.Generator(device="cuda").manual_seed(shift)
    rn = lambda m: torch.randn(m, device="cuda", generator=gen)
    k = torch.nn.functional.normalize(rn(layers * n * DK).view(-1, DK)).view(-1)
    v, g, beta = rn(layers * n * DK).bfloat16(), torch.exp(torch.nn.functional.logsigmoid(rn(layers * n * DK) + 3)), torch.sigmoid(rn(layers * n))
    states = rn(layers * len(rows) * per).to(torch.bfloat16 if state == "bf16" else torch.float32)
    cu = torch.tensor([0, 5, 7, 14, 17], dtype=torch.int32, device="cuda")
    kept = torch.tensor(keep, dtype=torch.int32, device="cuda")
    off = torch.arange(len(rows), dtype=torch.int64, device="cuda") * per
    moved = torch.zeros(v.numel() + 8, dtype=torch.bfloat16, device="cuda")
    moved[shift:shift + v.numel()] = v

    def run(vv, st):
        core.commit_batch(h, layers, cu, kept, st, len(rows) * per, off, (k, vv, g, beta), n * DK, n)
        return st

    got, want = run(moved[shift:], states.clone()), run(v, states.clone())
    torch.cuda.synchronize()
    assert torch.equal(got, want) and not torch.equal(got, states)
    names, _ = launches(lambda: run(moved[shift:], got))
    assert len(names) == 1 and "replay_small_kernel" in names[0], names


@pytest.mark.parametrize("state", ["f32", "bf16"])
@pytest.mark.parametrize("rows", [0, 1, 2, 3, 4, 5, 17])
def test_few_units_have_the_bits_of_many(rows, state):
    """Launches whose blocks find an SM each run replay_few_kernel: layer by layer the bits of all layers in one launch."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from captured import launches

    core = importlib.import_module("glm53f-afd_b200.core")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    h = 3 * sms // 16 if state == "f32" else sms // 4  # the most units that run there
    layers, n, per = 3, max(rows, 1) * h, h * DK * DK
    gen = torch.Generator(device="cuda").manual_seed(rows)
    rn = lambda m: torch.randn(m, device="cuda", generator=gen)
    k = torch.nn.functional.normalize(rn(layers * n * DK).view(-1, DK)).view(-1)
    v, g, beta = rn(layers * n * DK).bfloat16(), torch.exp(torch.nn.functional.logsigmoid(rn(layers * n * DK) + 3)), torch.sigmoid(rn(layers * n))
    states = rn(layers * per).to(torch.bfloat16 if state == "bf16" else torch.float32)
    cu, kept, off = (torch.tensor(x, dtype=d, device="cuda") for x, d in (([0, rows], torch.int32), ([rows], torch.int32), ([0], torch.int64)))

    def run(st, first, count):
        a, b = slice(first * n * DK, (first + count) * n * DK), slice(first * n, (first + count) * n)
        core.commit_batch(h, count, cu, kept, st[first * per:], per, off, (k[a], v[a], g[a], beta[b]), n * DK, n)

    many, few = states.clone(), states.clone()
    run(many, 0, layers)
    for layer in range(layers):
        run(few, layer, 1)
    torch.cuda.synchronize()
    assert torch.equal(many, few) and torch.equal(many, states) == (rows == 0)
    for count, kernel in ((1, "replay_few_kernel"), (layers, "replay_small_kernel")):
        names, _ = launches(lambda: run(few, 0, count))
        assert len(names) == 1 and kernel in names[0], names
