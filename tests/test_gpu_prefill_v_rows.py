"""Values behind a sequence's last row: the next sequence's are not numbers, as are the workspace's bytes, and neither reaches the sequence."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK = 128


@pytest.mark.parametrize("heads, chunks", [(4, 1), (4, 2), (4, 8), (80, 8)])  # halves by turns, side by side, all chunks, one launch
@pytest.mark.parametrize("rows", [1, 63, 64, 65, 130])
def test_core(heads, chunks, rows):
    core = importlib.import_module("glm53f-afd_b200.core")
    gen = torch.Generator(device="cuda").manual_seed(rows)
    total, per = rows + 64, heads * DK * DK
    n = total * heads
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    q, k, v = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16()
    g, beta = torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n))
    v[rows * heads * DK:] = float("nan")

    def run(lens):
        m = sum(lens) * heads
        st = torch.zeros(len(lens) * per, device="cuda")
        cu, off = torch.tensor([0] + lens, device="cuda").cumsum(0).int(), torch.arange(len(lens), device="cuda") * per
        out = torch.zeros(m * DK, dtype=torch.bfloat16, device="cuda")
        ws = torch.full((core.prefill_workspace_bytes(heads, len(lens), chunks),), 0xff, dtype=torch.uint8, device="cuda")
        core.prefill_varlen(heads, sum(lens), cu, max(lens), q[:m * DK], k[:m * DK], v[:m * DK], g[:m * DK], beta[:m], st, off, out=out, workspace=ws)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return out[:rows * heads * DK], st[:per]

    both, alone = run([rows, 64]), run([rows])
    for a, b in zip(both, alone):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("rows", [[65, 70, 1], [130, 64, 63]])
def test_layer(rows):
    K = importlib.import_module("glm53f-afd_b200.kernel")
    core = importlib.import_module("glm53f-afd_b200.core")
    h, gen = 64, torch.Generator(device="cuda").manual_seed(7)
    c, width, n, total = K.channels(h), h * DK, len(rows), sum(rows)
    rn = lambda m, s=1.0, d=torch.bfloat16: (torch.randn(m, device="cuda", generator=gen) * s).to(d)
    buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
    w = K.Weights(h, buf(rn(c * K.TAPS, 0.5)), buf(rn(h, 0.5, torch.float32)), buf(rn(width, 1.0, torch.float32)), buf(1 + rn(DK, 0.1)), 1e-5, -5.0)
    p, gates, conv = rn(total * (c + h)), rn(total * 2 * width), rn(n * 3 * c)
    form, got = K.set_prefill_form(K.Form.CHUNKED), []
    try:
        for fill in (0x00, 0xff):
            cv, state = conv.clone(), torch.zeros(n * K.state_len(h), device="cuda")
            out = torch.zeros(total * width, dtype=torch.bfloat16, device="cuda")
            ws = K.PrefillWorkspace.new(h, n, 256)
            ws.buf.t.fill_(fill)
            meta = K.BatchMeta.new(n)
            meta.set([K.Request(r, i * 3 * c, i * K.state_len(h)) for i, r in enumerate(rows)])
            g = buf(gates)
            K.PrefillBatch(w, K.RowView.dense(buf(p), c + h), c, K.RowView.new(g, 0, 2 * width), K.RowView.new(g, width, 2 * width), buf(cv), buf(state),
                           K.StateOut.InPlace, K.RowView.dense(buf(out), width), 0, ws).launch(meta, K.Stream())
            torch.cuda.synchronize()
            assert core.device_status() == 0
            got.append((out, state))
    finally:
        K.set_prefill_form(form)
    for a, b in zip(*got):
        assert torch.isfinite(a).all() and torch.equal(a, b)


def test_scan_over_segments(monkeypatch):
    core = importlib.import_module("glm53f-afd_b200.core")
    heads, lens, gen = 40, [300, 130], torch.Generator(device="cuda").manual_seed(5)
    n, per = sum(lens) * heads, heads * DK * DK
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    q, k, v = unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16()
    g, beta, start = torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n)), rn(2 * per) * 0.05
    cu, off = torch.tensor([0] + lens, device="cuda").cumsum(0).int(), torch.arange(2, device="cuda") * per

    def run(segments):
        monkeypatch.setenv("GLM53F_KDA_PREFILL_SEGMENTS", str(segments))
        out, st = torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda"), start.clone()
        ws = torch.full((core.prefill_workspace_bytes(heads, 2, 20),), 0xff, dtype=torch.uint8, device="cuda")
        core.prefill_varlen(heads, sum(lens), cu, max(lens), q, k, v, g, beta, st, off, out=out, workspace=ws)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return out.double(), st.double()

    (out, st), (out_1, st_1) = run(2), run(1)  # the bounds of the other scans: an ulp of bf16 of the largest output, the states' error of the chunked form
    assert float((out - out_1).abs().max() / out_1.abs().max()) <= 1 / 128
    assert 0 < float((st - st_1).norm() / st_1.norm()) <= 3e-4
