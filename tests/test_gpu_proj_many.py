"""Independent projections in one call against the same projections one by one, bit for bit (up to 512 rows; beyond, a shape
with a K split sums in one run on SM pairs both ways): row counts at the edges of both kernels' tiles, a K-split shape beside a
plain one, interleaved groups, ragged features and padded output rows that the tensor stores must leave alone."""
import ctypes as C
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 16, 17, 64, 65, 128, 129, 176, 177, 333, 512, 513, 700])
def test_many_equals_one_by_one(rows):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ffi = importlib.import_module("glm53f-afd_b200.ffi")
    lib, g = ffi.load(), torch.Generator(device="cuda").manual_seed(rows)
    mk = lambda *s: (torch.randn(*s, device="cuda", generator=g) * 0.1).bfloat16()
    # (groups, n, k, padding of the output rows): a K split, ragged features, two groups interleaved in the output rows
    shapes = [(1, 256, 2048, 0), (1, 1112, 512, 8), (2, 264, 128, 0)]
    jobs, outs = [], []
    for groups, n, k, pad in shapes:
        x, w = mk(rows, groups * k), mk(groups, n, k)
        ldo = groups * n + pad
        pair = [torch.full((rows * ldo + 64,), 3.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        outs.append((pair, groups * n, ldo, x, w))
        jobs.append([ffi.ProjJob(x.data_ptr(), groups * k, k, w.data_ptr(), k, n * k, groups, rows, n, k, o.data_ptr(), 0, ldo, n) for o in pair])
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.glm53f_kda_proj_bf16_many((ffi.ProjJob * 3)(*[j[0] for j in jobs]), 3, stream) == 0
    for j in jobs:
        assert lib.glm53f_kda_proj_bf16(*(getattr(j[1], f) for f, _ in ffi.ProjJob._fields_), stream) == 0
    torch.cuda.synchronize()
    for (a, b), width, ldo, x, w in outs:
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
        body = a[:rows * ldo].view(rows, ldo)
        assert (body[:, width:] == 3.0).all() and (a[rows * ldo:] == 3.0).all()
        groups, n, k = w.shape
        want = torch.einsum("rgk,gnk->rgn", x.view(rows, groups, k).double(), w.double()).reshape(rows, -1)
        # f32 sums of k products, then one rounding to bf16 (2^-9 of the value)
        assert ((body[:, :width].double() - want).abs() <= want.abs() * 2 ** -8 + k ** 0.5 * 1e-6).all()
    bad = (ffi.ProjJob * 2)(jobs[0][0], jobs[1][0])
    bad[1].k = 100
    assert lib.glm53f_kda_proj_bf16_many(bad, 2, stream) == 1  # checked before anything is launched


@pytest.mark.parametrize("rows", [1, 16, 17, 32, 33, 64, 65, 96])
@pytest.mark.parametrize("shapes", [[(1, 256, 1024), (1, 1112, 1024)], [(1, 9608, 512), (1, 264, 512)], [(2, 4808, 128), (1, 9600, 256)], [(1, 256, 4096), (1, 9600, 4096)]])
def test_few_rows_share_a_launch(rows, shapes):
    """Two GEMMs of few rows whose tiles share a launch, and one that has to stay apart (both split): with a split k (its parts summed by one block then),
    without, ragged features and rows; the bits of each alone."""
    ffi = importlib.import_module("glm53f-afd_b200.ffi")
    lib, g = ffi.load(), torch.Generator(device="cuda").manual_seed(rows)
    mk = lambda *s: (torch.randn(*s, device="cuda", generator=g) * 0.1).bfloat16()
    jobs, outs, keep = [], [], []
    for f32, (groups, n, k) in enumerate(shapes):
        x, w = mk(rows, groups * k), mk(groups, n, k)
        ldo, kind = groups * n + 8, torch.float32 if f32 else torch.bfloat16
        pair = [torch.full((rows * ldo + 64,), 3.0, dtype=kind, device="cuda") for _ in range(2)]
        keep.append((x, w))
        outs.append(pair)
        jobs.append([ffi.ProjJob(x.data_ptr(), groups * k, k, w.data_ptr(), k, n * k, groups, rows, n, k, o.data_ptr(), f32, ldo, n) for o in pair])
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.glm53f_kda_proj_bf16_many((ffi.ProjJob * 2)(*[j[0] for j in jobs]), 2, stream) == 0
    for j in jobs:
        assert lib.glm53f_kda_proj_bf16(*(getattr(j[1], f) for f, _ in ffi.ProjJob._fields_), stream) == 0
    torch.cuda.synchronize()
    assert importlib.import_module("glm53f-afd_b200.core").device_status() == 0
    for a, b in outs:
        assert torch.equal(a, b)
