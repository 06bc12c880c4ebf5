"""GLM53F_KDA_PDL=0 makes every launch of the library a plain one: a step of each kind is captured in a process of its own (the variable
is read once), and no launch in it may begin before its predecessor has ended.  Without the variable they may."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

STEP = r"""
import importlib, sys
import torch
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
from captured import launches
core, K, proj = (importlib.import_module("glm53f-afd_b200." + m) for m in ("core", "kernel", "proj"))
DK, h, slots, rows = 128, 4, 2, 3
n, total, c, width, per = slots * rows * h, slots * rows, K.channels(h), h * DK, K.state_len(h)
zb = lambda m: torch.zeros(m, dtype=torch.bfloat16, device="cuda")
zf = lambda m: torch.zeros(m, device="cuda")
buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
w = K.Weights(h, buf(zb(c * 4)), buf(zf(h)), buf(zf(width)), buf(zb(DK)), 1e-5, -5.0)
stride = c + 64
p, gates, conv, out, state = buf(zb(total * stride)), buf(zb(total * 2 * width)), buf(zb(slots * 3 * c)), buf(zb(total * width)), buf(zb(slots * per))
views = (K.RowView.dense(p, stride), c, K.RowView.new(gates, 0, 2 * width), K.RowView.new(gates, width, 2 * width))
meta = K.BatchMeta.new(slots)
meta.set([K.Request(rows, i * 3 * c, i * per) for i in range(slots)])
saves = (zf(n * DK), zb(n * DK), zf(n * DK), zf(n))
q, o, g, beta, st = zb(n * DK), zb(n * DK), zf(n * DK), zf(n), zb(slots * per)
cu, off = torch.tensor([0, 3, 6], dtype=torch.int32, device="cuda"), torch.tensor([0, per], dtype=torch.int64, device="cuda")
keep = torch.tensor([2, 1], dtype=torch.int32, device="cuda")
x, weight, y = zb(2048 * 256), proj.Bf16Mat.dense(zb(256 * 256).view(256, 256)), zb(2048 * 256)
prefill = K.PrefillBatch(w, *views, conv, state, K.StateOut.InPlace, K.RowView.dense(out, width), 0, K.PrefillWorkspace.new(h, slots, 64))
decode = K.ChainBatch(w, *views, conv, state, K.StateOut.InPlace, K.RowView.dense(out, width))
verify = K.ChainBatch(w, *views, conv, state, K.StateOut.Skip, K.RowView.dense(out, width), K.Saves.alloc(h, total))
ws = torch.empty(core.prefill_workspace_bytes(h, slots, 4), dtype=torch.uint8, device="cuda")


def step():
    s = K.Stream()
    for flags, form in ((0, K.Form.EXACT), (core.TENSOR, K.Form.CHUNKED)):
        K.set_commit_form(form)
        K.set_prefill_form(form)
        K.set_verify_form(form)
        verify.launch_bf16_state(meta, s)
        core.decode_batch(h, total, cu, q, q, q, g, beta, st, off, state_out=None, flags=flags, out=o, saves=saves)
        core.commit_batch(h, 1, cu, keep, st, slots * per, off, saves, n * DK, n)
        prefill.launch_bf16_state(meta, s)
    core.decode_batch(h, total, cu, q, q, q, g, beta, st, off, out=o)
    decode.launch_bf16_state(meta, s)
    K.conv_shift_batch(h, 1, meta, conv, slots * 3 * c, views[0], total * stride, s)
    for scratch in (None, ws):
        core.prefill_varlen(h, total, cu, rows, q, q, q, g, beta, st, off, out=o, workspace=scratch)
    for r in (16, 2048):
        proj.bf16(x, 256, 0, weight, r, y, 256, 0)


step()
assert core.device_status() == 0
names, early = launches(step)
print(len(names), early)
"""


@pytest.mark.parametrize("plain", [True, False])
def test_the_switch_reaches_every_launch(plain):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = {k: v for k, v in os.environ.items() if k != "GLM53F_KDA_PDL"}
    if plain:
        env["GLM53F_KDA_PDL"] = "0"
    r = subprocess.run([sys.executable, "-c", STEP, root], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    launched, early = map(int, r.stdout.split()[-2:])
    assert launched >= 18
    assert early == 0 if plain else early > 10
