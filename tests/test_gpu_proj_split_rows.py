"""Shapes of few features, whose small launches add k in parts, in launches of more than 512 rows: the same parts in the same order,
so every row has the bits of a launch of 64 rows.  Row counts at the edges of the segmented tiles (144, 160, 192 and 128 rows for
o_proj's shape, 16 for the first gate factor's)."""
import ctypes as C
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, k, rows", [(4096, 8192, 513), (4096, 8192, 640), (4096, 8192, 641), (4096, 8192, 768), (4096, 8192, 769), (4096, 8192, 1024),
                                        (256, 4096, 513), (256, 4096, 1184), (256, 4096, 1185), (256, 4096, 2048)])
def test_rows_keep_the_bits_of_small_launches(n, k, rows):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ffi = importlib.import_module("glm53f-afd_b200.ffi")
    lib, g = ffi.load(), torch.Generator(device="cuda").manual_seed(rows)
    x, w = ((torch.randn(m, k, device="cuda", generator=g) * 0.1).bfloat16() for m in (rows, n))
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def run(first, count):
        out = torch.zeros(count, n, device="cuda")
        assert lib.glm53f_kda_proj_bf16(x[first:].data_ptr(), k, 0, w.data_ptr(), k, 0, 1, count, n, k, out.data_ptr(), 1, n, 0, stream) == 0
        return out

    whole = run(0, rows)
    for first in range(0, rows, 64):
        count = min(64, rows - first)
        assert torch.equal(whole[first:first + count].view(torch.int32), run(first, count).view(torch.int32)), first
