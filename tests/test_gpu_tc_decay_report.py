"""Seven rows behind a window's middle row that decay by more than 2^-126: what cannot be split into factors is reported (status 121) by the
chunked commit, for rows that are kept, and by the layer form of the chunked verify, whose decay factors come from saved multipliers too."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
H, ROWS, DK = 4, 16, 128


@pytest.fixture(scope="module")
def G():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import kda_gpu

    kda_gpu.product()
    return kda_gpu


def status(G):
    torch.cuda.synchronize()
    return G.ffi.load().glm53f_kda_device_status()


@pytest.fixture()
def window(G, oracle):
    o = oracle
    p, rows = o.Layer(H, 411), o.Rows(H, ROWS, 411)
    rows.a[:] = np.where(np.arange(rows.a.size) // (H * DK) >= 9, 1e4, -1e4)  # rows 9 to 15 at the lower bound, the others do not decay
    return p, o.conv_window(H, 411), o.bf16_round_np(o.state(H, 411, 0.5)), rows


@pytest.mark.parametrize("lower, keep, want", [(-10.5, 16, 0), (-12.0, 16, 0), (-13.0, 16, 121), (-13.0, 9, 0), (-13.0, 15, 0), (-15.0, 15, 121)])
def test_commit(G, oracle, window, lower, keep, want):
    lib, (p, conv, s0, rows) = G.product(), window
    p.lower = lower
    sv = G.run_chain(lib, p, conv, s0, rows, bf16_state=True, write_state=False)
    before = lib.glm53f_kda_commit_mode(1)
    try:
        got = G.run_replay(lib, H, s0, sv, keep, bf16_state=True)
    finally:
        lib.glm53f_kda_commit_mode(before)
    assert status(G) == want and status(G) == 0
    assert np.isfinite(got).all()
    if want == 0:
        # One bf16 rounding of the state is 1.7e-3 of its norm, the bf16 operands add less.  (Not against the exact replay, which rounds after
        # every row: nine rows that do not decay are sqrt(9) x 1.7e-3 = 5e-3 from the recurrence by themselves.)
        assert G.rel_l2(got, oracle.replay(s0, sv, keep, bf16_state=False)) <= 3e-3


@pytest.mark.parametrize("lower, want", [(-10.5, 0), (-12.0, 0), (-13.0, 121)])
def test_layer_verify(G, window, lower, want):
    lib, (p, conv, s0, rows) = G.product(), window
    p.lower = lower
    exact = G.run_chain(lib, p, conv, s0, rows, bf16_state=True, write_state=False)
    before = lib.glm53f_kda_verify_mode(1)
    try:
        got = G.run_chain(lib, p, conv, s0, rows, bf16_state=True, write_state=False)
    finally:
        lib.glm53f_kda_verify_mode(before)
    assert got.rc == 0
    assert status(G) == want and status(G) == 0
    assert np.isfinite(got.out).all()
    if lower == -10.5:  # the bound of the other chunked verifies (at e^-84 a factor's bf16 operands are denormal)
        assert G.rel_l2(got.out, exact.out) <= 1e-2
