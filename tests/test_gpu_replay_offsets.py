"""The commit replay whose saved values start at any element: those on 8 bytes run on the small-block kernel (csrc/kda_chain.cu,
replay_entry), the others on the persistent one, with the same bits.  Prefix lengths around the rows kept in flight."""
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
