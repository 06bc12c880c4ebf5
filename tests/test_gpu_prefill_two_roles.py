"""The two roles over a workspace at lengths that a call which names them would run without it: a longer longest sequence than there is takes them.  Heads
on both sides of the line from which on the walk forms U, and as many chains as make one launch of it."""
import importlib
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DK, LONG = 128, 64 * 64
core = importlib.import_module("glm53f-afd_b200.core")


def rows_of(n, gen):
    """q, k, v, the log decays and beta of n rows and heads"""
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    unit = lambda s: torch.nn.functional.normalize(rn(n, DK), dim=1).mul(s).bfloat16().view(-1)
    return unit(DK ** -0.5), unit(1.0), rn(n * DK).bfloat16(), torch.nn.functional.logsigmoid(rn(n * DK) + 3), torch.sigmoid(rn(n))


def prefill(heads, lens, rows, states, workspace, **extra):
    per, n = heads * DK * DK, sum(lens) * heads
    out, st = torch.zeros(n * DK, dtype=torch.bfloat16, device="cuda"), states.clone()
    cu, off = torch.tensor([0] + lens, device="cuda").cumsum(0).int(), torch.arange(len(lens), device="cuda") * per
    core.prefill_varlen(heads, sum(lens), cu, LONG, *rows, st, off, out=out, workspace=workspace, **extra)
    torch.cuda.synchronize()
    return out, st


def workspace(heads, batch, chunks):
    return torch.full((core.prefill_workspace_bytes(heads, batch, chunks),), 0xff, dtype=torch.uint8, device="cuda")


def recurrence(q, k, v, g, beta, s):
    """64 bits; [rows][heads][128], state [head][value][key]"""
    q, k, v, e, beta, out = q.double(), k.double(), v.double(), g.double().exp(), beta.double(), []
    for t in range(q.shape[0]):
        s = s * e[t][:, None, :]
        s = s + (beta[t][:, None] * (v[t] - (s * k[t][:, None, :]).sum(-1)))[:, :, None] * k[t][:, None, :]
        out.append((s * q[t][:, None, :]).sum(-1))
    return torch.stack(out), s


@pytest.mark.parametrize("chunks", [1, 2, 8])
@pytest.mark.parametrize("heads", [4, 40, 80])
@pytest.mark.parametrize("rows", [1, 63, 64, 65, 130])
def test_behind_the_last_row(heads, chunks, rows):
    """The next sequence's values and the workspace's bytes are not numbers, and neither reaches a sequence: its bits are those that it has alone."""
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x, per, m = rows_of((rows + 64) * heads, gen), heads * DK * DK, rows * heads
    x[2][m * DK:] = float("nan")
    out, st = prefill(heads, [rows, 64], x, torch.zeros(2 * per, device="cuda"), workspace(heads, 2, chunks))
    alone = prefill(heads, [rows], [t[:m * (1 if t.numel() == (rows + 64) * heads else DK)].clone() for t in x], torch.zeros(per, device="cuda"), workspace(heads, 1, chunks))
    assert core.device_status() == 0
    for a, b in zip((out[:m * DK], st[:per]), alone):
        same = bool(torch.isfinite(a).all()) and torch.equal(a, b)
        assert same


@pytest.mark.parametrize("heads", [2, 40, 160])
@pytest.mark.parametrize("decay", [-5.8, -6.2])
def test_steep_blocks(decay, heads):
    """A block of sixteen rows decays past the smallest normal number, its first row repeats the last one before it and does not decay: the pair's factor e^0 is
    e^+46 x e^-93 x e^+47.  The bounds of the same rows by the other kernel: 1e-2 of the norm for bf16 operands, a lost pair is 0.9 of its row."""
    n, gen = 128, torch.Generator(device="cuda").manual_seed(5)
    q, k, v, _, _ = (t.view(n, heads, -1) for t in rows_of(n * heads, gen))
    k[16::16], q[16::16] = k[15:-1:16].clone(), q[15:-1:16].clone()
    g, beta = torch.full((n, heads, DK), decay, device="cuda"), torch.full((n, heads), 0.9, device="cuda")
    g[16::16] = -0.01
    want, s = recurrence(q, k, v, g, beta, torch.zeros(heads, DK, DK, dtype=torch.float64, device="cuda"))
    out, st = prefill(heads, [n], [t.reshape(-1) for t in (q, k, v, g, beta)], torch.zeros(heads * DK * DK, device="cuda"), workspace(heads, 1, 2))
    assert core.device_status() == 0
    assert (out.view(n, heads, DK).double() - want).norm() <= 1e-2 * want.norm()
    assert (st.view(heads, DK, DK).double() - s).norm() <= 2e-3 * s.norm()


@pytest.mark.parametrize("heads, scratch", [(2, "workspace"), (2, "static"), (40, "workspace"), (160, "workspace")])
@pytest.mark.parametrize("first, last, decay, status", [(9, 16, -12.0, 0), (9, 16, -13.0, 121), (0, 70, -12.0, 121), (0, 70, -5.8, 0)])
def test_decay_that_cannot_be_split(heads, scratch, first, last, decay, status):
    n, gen = 70, torch.Generator(device="cuda").manual_seed(6)
    x = rows_of(n * heads, gen)
    g = x[3].view(n, -1)
    g[:] = -0.1
    g[first:last] = decay
    out, st = prefill(heads, [n], x, torch.zeros(heads * DK * DK, device="cuda"), workspace(heads, 1, 2) if scratch == "workspace" else scratch)
    assert core.device_status() == status
    assert core.device_status() == 0
    if first == 9:  # (factors of eight rows before a middle row are past the largest number)
        finite = bool(torch.isfinite(out).all())
        assert finite


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("heads, rows", [(64, 4033), (64, 8129), (40, 8160)])  # 64 and 128 chunks, the last ones partial: two and three parts
def test_parts_where_the_walk_forms_u(heads, rows, fused):
    """A workspace that holds the whole call is used in parts; the results are those of a small one."""
    gen = torch.Generator(device="cuda").manual_seed(rows)
    x, states = rows_of(rows * heads, gen), torch.randn(heads * DK * DK, device="cuda", generator=gen) * 0.05
    extra = {"gate": torch.randn(rows * heads * DK, device="cuda", generator=gen).bfloat16(), "norm_w": torch.ones(DK, dtype=torch.bfloat16, device="cuda")} if fused else {}

    def run(chunks):
        per = heads * DK * DK
        out, st = torch.zeros(rows * heads * DK, dtype=torch.bfloat16, device="cuda"), states.clone()
        core.prefill_varlen(heads, rows, torch.tensor([0, rows], dtype=torch.int32, device="cuda"), rows, *x, st, torch.zeros(1, dtype=torch.int64, device="cuda"), out=out,
                            workspace=workspace(heads, 1, chunks), **extra)
        torch.cuda.synchronize()
        assert core.device_status() == 0
        return out, st

    for a, b in zip(run(300), run(10)):
        same = bool(torch.isfinite(a).all()) and torch.equal(a, b)
        assert same


STEP = r"""
import importlib, sys
import torch
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
from captured import launches
core = importlib.import_module("glm53f-afd_b200.core")
zb, zf = lambda m: torch.zeros(m, dtype=torch.bfloat16, device="cuda"), lambda m: torch.zeros(m, device="cuda")
calls = []
for h in (4, 40, 160):
    n = 3 * h
    calls.append((h, 3, torch.tensor([0, 3], dtype=torch.int32, device="cuda"), 256, zb(n * 128), zb(n * 128), zb(n * 128), zf(n * 128), zf(n), zf(h * 128 * 128),
                  torch.zeros(1, dtype=torch.int64, device="cuda")))
keep = [(zb(3 * c[0] * 128), torch.empty(core.prefill_workspace_bytes(c[0], 1, 4), dtype=torch.uint8, device="cuda")) for c in calls]


def step():
    for c, (out, ws) in zip(calls, keep):
        core.prefill_varlen(*c, out=out, workspace=ws)


step()
assert core.device_status() == 0
names, early = launches(step)
print(len(names), early)
"""


@pytest.mark.parametrize("plain", [True, False])
def test_the_switch_of_plain_launches(plain):
    """GLM53F_KDA_PDL=0, read once a process: no launch may begin before its predecessor has ended.  (Two segments are three launches, twice, and a pass with
    more chains than SMs is one.)"""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = {k: v for k, v in os.environ.items() if k != "GLM53F_KDA_PDL"}
    if plain:
        env["GLM53F_KDA_PDL"] = "0"
    r = subprocess.run([sys.executable, "-c", STEP, root], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    launched, early = map(int, r.stdout.split()[-2:])
    assert launched == 7
    assert early == 0 if plain else early > 0
