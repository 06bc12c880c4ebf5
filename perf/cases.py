"""The work that users of this library have it do, as cases that can be timed and compared.

A case is one step of a serving engine on the KDA layers of the model (34 layers of 64 heads, 128 x 128 states): the
calls a program makes for that step, on buffers it keeps.  Kinds:

  decode_layer   one token for each slot through every layer: `ChainBatch` on projection rows, then the conv windows' shift
  decode_core    the same on post-convolution inputs (`core.decode_batch`)
  verify_layer   a round of draft verification over pool slots (`KdaVerify`): open, every layer, commit of a prefix
  verify_core    the round on post-convolution inputs: `core.decode_batch` with saves per layer, one `core.commit_batch`
  prefill_layer  a prompt segment of each lane through one layer (`PrefillBatch`)
  prefill_core   packed sequences through one layer's chunked prefill (`core.prefill_varlen`)
  proj           the four GEMMs of one layer: the input projections and the output projection
  mark           snapshot of each slot's positional state into pool pages and its restore into another slot

`form` is the library's switch between the exact kernels ("exact": results bit for bit those of serial single-row steps)
and the tensor-core ones ("chunked": results to the rounding of bf16 operands).
"""
from __future__ import annotations

import importlib
import math
import random

import torch

_PKG = "glm53f-afd_b200"
core = importlib.import_module(_PKG + ".core")
K = importlib.import_module(_PKG + ".kernel")
marks = importlib.import_module(_PKG + ".marks")
proj = importlib.import_module(_PKG + ".proj")
verify = importlib.import_module(_PKG + ".verify")

LAYERS, HEADS, DK = 34, 64, 128
CONV = 3 * HEADS * DK                    # conv channels q | k | v
P_COLS = CONV + HEADS                    # a projection row: q | k | v | beta logits
WIDTH = HEADS * DK
STATE = HEADS * DK * DK                  # elements of one layer's state
ROW_CORE = DK * 12 + 4                   # bytes of one row and head: q, k, v, out bf16, log decay f32, beta f32
ROW_SAVES = DK * 10 + 4                  # k and decay f32, v bf16, beta f32
ROW_LAYER = 2 * (P_COLS + 3 * WIDTH)     # a layer row: projections, both gates, the output
WINDOW_BYTES = 2 * K.WINDOW * CONV       # one slot's conv window
WEIGHT_BYTES = 2 * K.TAPS * CONV + 4 * (HEADS + WIDTH) + 2 * DK


def listed():
    return [
        # The smallest step there is: one user, one token, the model's 34 layers; launches and host work count here.
        {"name": "decode_1_slot", "kind": "decode_layer", "slots": 1, "state": "bf16"},
        # The ordinary decode step of a busy server (the benchmark's default workload: 16 slots, bf16 states).
        {"name": "decode_16_slots", "kind": "decode_core", "slots": 16, "state": "bf16"},
        # A speculative round of a few users on full-precision states, ragged windows, through the orchestration.
        {"name": "verify_round_6_slots", "kind": "verify_layer", "slots": 6, "window": 8, "state": "f32", "form": "exact"},
        # The benchmark's draft verification: 48 slots x 16 rows, the tensor-core forms of verify and commit.
        {"name": "verify_48_slots", "kind": "verify_core", "slots": 48, "window": 16, "state": "bf16", "form": "chunked"},
        # A short prompt through the default form of the layer prefill (bit for bit the serial steps).
        {"name": "prompt_exact_701", "kind": "prefill_layer", "lanes": 1, "rows": 701, "state": "f32", "form": "exact", "pass_rows": 256},
        # The coordinator's prefill: four lanes of 2,048 rows, the tensor-core form, the default workspace.
        {"name": "prompt_lanes_4x2048", "kind": "prefill_layer", "lanes": 4, "rows": 2048, "state": "bf16", "form": "chunked", "pass_rows": 256},
        # Packed prompts of unequal length, half of them continuing a carried state, with a workspace.
        {"name": "packed_8192", "kind": "prefill_core", "heads": 64, "sequences": 8, "rows": 8192, "state": "f32", "chunks": 32, "fused": False},
        # A long document: one sequence, 64 chains only.
        {"name": "long_262144", "kind": "prefill_core", "heads": 64, "sequences": 1, "rows": 262144, "state": "f32", "chunks": 256, "fused": False},
        # The GEMMs around the core for a decode step, a ragged verify or prompt tail, and a prefill lane.
        {"name": "projections_16", "kind": "proj", "rows": 16},
        {"name": "projections_333", "kind": "proj", "rows": 333},
        {"name": "projections_2048", "kind": "proj", "rows": 2048},
        # Prefix-cache hits: each of four slots is snapshotted and another slot forked from the snapshot.
        {"name": "mark_fork_4", "kind": "mark", "slots": 4, "state": "bf16"},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(("decode_layer", "decode_layer", "decode_core", "decode_core", "verify_layer", "verify_layer",
                       "verify_core", "verify_core", "prefill_layer", "prefill_layer", "prefill_core", "prefill_core", "proj", "proj", "proj", "mark"))
    state, form = rng.choice(("bf16", "f32")), rng.choice(("exact", "chunked"))
    if kind == "decode_layer":
        return {"kind": kind, "slots": _log(rng, 3, 48), "state": state}
    if kind == "decode_core":
        return {"kind": kind, "slots": _log(rng, 2, 64), "state": state}
    if kind == "verify_layer":
        return {"kind": kind, "slots": _log(rng, 2, 12), "window": rng.randint(2, 8), "state": state, "form": form}
    if kind == "verify_core":
        return {"kind": kind, "slots": _log(rng, 2, 40), "window": rng.randint(3, 16), "state": "bf16", "form": form}
    if kind == "prefill_layer":
        return {"kind": kind, "lanes": rng.randint(1, 4), "rows": _log(rng, 65, 2048), "state": state, "form": form, "pass_rows": rng.choice((256, 1024))}
    if kind == "prefill_core":
        sequences = rng.randint(1, 8)
        return {"kind": kind, "heads": rng.choice((8, 16, 32, 64, 64)), "sequences": sequences, "rows": _log(rng, 96 * sequences, 98304),
                "state": state, "chunks": rng.choice((0, 32, 256)), "fused": rng.random() < 0.3}
    if kind == "proj":
        return {"kind": kind, "rows": _log(rng, 1, 4096)}
    return {"kind": kind, "slots": rng.choice((1, 2, 3, 5, 6, 7, 8)), "state": state}


# ---- what the sizes of a case imply -----------------------------------------------------------------------------

def _windows(case):
    """Rows of each slot's draft window and the accepted prefix: ragged, the same for every seed."""
    r = random.Random(1000 * case["slots"] + case["window"])
    rows = [r.randint(max(1, case["window"] // 2), case["window"]) for _ in range(case["slots"])]
    return rows, [r.randint(1, n) for n in rows]


def _lengths(case):
    """Lengths of the packed sequences: unequal, at least one row each, summing to the case's rows."""
    r = random.Random(case["rows"] * 31 + case["sequences"])
    share = [r.uniform(0.35, 1.0) for _ in range(case["sequences"])]
    at = [round(sum(share[:i]) / sum(share) * case["rows"]) for i in range(case["sequences"] + 1)]
    return [b - a for a, b in zip(at, at[1:])]


def _state_bytes(case):
    return 2 if case["state"] == "bf16" else 4


def _layout(case):
    return marks.KvLayout.glm53_flash().with_kda_state_bf16(case["state"] == "bf16")


def work(case):
    """Bytes: each input read once and each output written once.  Operations of a row and head: the recurrence's 7 per
    state element (decay, read-out of k, update, read-out of q), or the causal chunk-64 form's for a prefill."""
    kind, step = case["kind"], 7 * DK * DK
    if kind in ("decode_layer", "decode_core"):
        s = case["slots"]
        row = ROW_LAYER + 2 * WINDOW_BYTES if kind == "decode_layer" else HEADS * ROW_CORE
        fixed = WEIGHT_BYTES if kind == "decode_layer" else 0
        return {"bytes": LAYERS * (s * (2 * STATE * _state_bytes(case) + row) + fixed), "flops": LAYERS * s * HEADS * step}
    if kind in ("verify_layer", "verify_core"):
        rows, keep = _windows(case)
        r, k, s = sum(rows), sum(keep), case["slots"]
        row = ROW_LAYER if kind == "verify_layer" else HEADS * ROW_CORE
        fixed = WEIGHT_BYTES + 2 * s * WINDOW_BYTES if kind == "verify_layer" else 0
        # the states are read for the outputs, then read and written by the commit; the kept rows' saves are read back
        return {"bytes": LAYERS * (3 * s * STATE * _state_bytes(case) + r * row + (r + k) * HEADS * ROW_SAVES + fixed),
                "flops": LAYERS * (r + k) * HEADS * step}
    if kind == "prefill_layer":
        r, s = case["lanes"] * case["rows"], case["lanes"]
        flops = HEADS * step if case["form"] == "exact" else 8.94e6
        return {"bytes": r * ROW_LAYER + s * (2 * STATE * _state_bytes(case) + 2 * WINDOW_BYTES) + WEIGHT_BYTES, "flops": r * flops}
    if kind == "prefill_core":
        r, h = case["rows"], case["heads"]
        return {"bytes": r * h * (ROW_CORE + (2 * DK if case["fused"] else 0)) + 2 * case["sequences"] * h * DK * DK * _state_bytes(case),
                "flops": r * h * 8.94e6 / 64}
    if kind == "proj":
        r = case["rows"]
        weights = [(P_COLS, proj.HIDDEN), (2 * DK, proj.HIDDEN), (2 * WIDTH, DK), (proj.HIDDEN, WIDTH)]
        return {"bytes": 2 * sum(n * k for n, k in weights) + 2 * r * (proj.HIDDEN + P_COLS + 2 * DK + 2 * WIDTH + WIDTH + proj.HIDDEN),
                "flops": 2 * r * sum(n * k for n, k in weights)}
    return {"bytes": 4 * case["slots"] * _layout(case).mark_bytes(), "flops": 0}  # snapshot, then restore


def tolerance(case):
    """The exact forms and the copies promise their bits.  A tensor-core form rounds its operands to bf16 and its outputs
    too; a projection only rounds its f32 sums to bf16 (the second gate factor takes rounded inputs)."""
    if case["kind"] in ("decode_layer", "decode_core", "mark"):
        return "exact"
    if case["kind"] == "proj":
        return {"rel": 4e-3}
    if case["kind"] == "prefill_core" or case["form"] == "chunked":
        return {"rel": 1e-2}
    return "exact"


# ---- inputs -----------------------------------------------------------------------------------------------------

class _Gen:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(0x53454544 + seed)

    def normal(self, n, std=1.0, dtype=torch.bfloat16, mean=0.0, piece=1 << 28):
        out = torch.empty(n, dtype=dtype, device="cuda")
        for a in range(0, n, piece):  # in pieces: bounds the f32 temporaries
            m = min(piece, n - a)
            out[a:a + m] = torch.randn(m, device="cuda", generator=self.g).mul_(std).add_(mean)
        return out

    def unit(self, rows, scale, piece=1 << 21):
        """Rows of 128, L2-normalised, times `scale`, bf16."""
        out = torch.empty(rows, DK, dtype=torch.bfloat16, device="cuda")
        for a in range(0, rows, piece):
            m = min(piece, rows - a)
            x = torch.randn(m, DK, device="cuda", generator=self.g)
            out[a:a + m] = x.mul_(scale / torch.sqrt((x * x).sum(1, keepdim=True) + 1e-6))
        return out.view(-1)

    def log_decay(self, n, piece=1 << 28):
        out = torch.empty(n, device="cuda")
        for a in range(0, n, piece):
            m = min(piece, n - a)
            out[a:a + m] = torch.nn.functional.logsigmoid(torch.randn(m, device="cuda", generator=self.g).add_(3.0))
        return out

    def tokens(self, rows, heads=HEADS):
        """Post-convolution inputs of `rows` rows: q, k, v, log decay, beta."""
        n = rows * heads
        return (self.unit(n, DK ** -0.5), self.unit(n, 1.0), self.normal(n * DK), self.log_decay(n * DK),
                torch.sigmoid(torch.randn(n, device="cuda", generator=self.g)))

    def states(self, n, kind):
        return self.normal(n, 0.05, torch.bfloat16 if kind == "bf16" else torch.float32)

    def weights(self):
        """One layer's weights on the device."""
        buf = lambda t: K.DeviceBuffer(t.view(torch.uint8))
        return K.Weights(HEADS, buf(self.normal(CONV * K.TAPS, 0.5)), buf(self.normal(HEADS, 0.5, torch.float32)), buf(self.normal(WIDTH, 1.0, torch.float32)),
                         buf(self.normal(DK, 0.1, mean=1.0)), 1e-5, -5.0)


def _bytes(t):
    return K.DeviceBuffer(t.view(torch.uint8))


def _cu(lengths):
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    return torch.tensor(cu, dtype=torch.int32, device="cuda")


def _offsets(n, per):
    return torch.arange(n, dtype=torch.int64, device="cuda") * per


def _prepare_decode_layer(case, gen):
    slots, elem = case["slots"], _state_bytes(case)
    s = {"stream": K.Stream(), "weights": [gen.weights() for _ in range(LAYERS)]}
    s["p"], s["gates"] = gen.normal(LAYERS * slots * P_COLS), gen.normal(LAYERS * slots * 2 * WIDTH)
    s["conv"], s["state"] = gen.normal(LAYERS * slots * 3 * CONV), gen.states(LAYERS * slots * STATE, case["state"])
    s["out"] = torch.zeros(LAYERS * slots * WIDTH, dtype=torch.bfloat16, device="cuda")
    s["meta"] = K.BatchMeta.new(slots)
    s["meta"].set([K.Request(1, i * 3 * CONV, i * STATE) for i in range(slots)])
    p, gates, conv, state, out = (_bytes(s[n]) for n in ("p", "gates", "conv", "state", "out"))
    part = lambda b, at, n: K.DeviceBuffer(b.t[at:at + n])
    s["layers"] = [
        K.ChainBatch(s["weights"][j], K.RowView.new(p, j * slots * P_COLS, P_COLS), CONV, K.RowView.new(gates, j * slots * 2 * WIDTH, 2 * WIDTH),
                     K.RowView.new(gates, j * slots * 2 * WIDTH + WIDTH, 2 * WIDTH), part(conv, j * slots * 3 * CONV * 2, slots * 3 * CONV * 2),
                     part(state, j * slots * STATE * elem, slots * STATE * elem), K.StateOut.InPlace, K.RowView.new(out, j * slots * WIDTH, WIDTH))
        for j in range(LAYERS)]
    s["conv_buf"], s["p_rows"] = conv, K.RowView.new(p, 0, P_COLS)
    return s


def _run_decode_layer(case, s):
    meta, stream, slots = s["meta"], s["stream"], case["slots"]
    for cb in s["layers"]:
        if case["state"] == "bf16":
            cb.launch_bf16_state(meta, stream)
        else:
            cb.launch(meta, stream)
    K.conv_shift_batch(HEADS, LAYERS, meta, s["conv_buf"], slots * 3 * CONV, s["p_rows"], slots * P_COLS, stream)
    return s["out"], s["state"], s["conv"]


def _prepare_decode_core(case, gen):
    slots = case["slots"]
    s = {"layers": [gen.tokens(slots) for _ in range(LAYERS)], "cu": _cu([1] * slots), "off": _offsets(slots, STATE)}
    s["state"] = gen.states(LAYERS * slots * STATE, case["state"])
    s["states"] = list(s["state"].view(LAYERS, -1))
    s["out"] = torch.zeros(LAYERS, slots * WIDTH, dtype=torch.bfloat16, device="cuda")
    s["outs"] = list(s["out"])
    return s


def _run_decode_core(case, s):
    for (q, k, v, g, beta), state, out in zip(s["layers"], s["states"], s["outs"]):
        core.decode_batch(HEADS, case["slots"], s["cu"], q, k, v, g, beta, state, s["off"], out=out)
    return s["out"], s["state"]


def _prepare_verify_layer(case, gen):
    rows, keep = _windows(case)
    total, slots = sum(rows), case["slots"]
    pool = marks.KvPool(marks.KvConfig(_layout(case), slots, 1))
    kvs = [pool.slot() for _ in range(slots)]
    pool.state.t.view(torch.bfloat16 if case["state"] == "bf16" else torch.float32).copy_(gen.states(slots * LAYERS * STATE, case["state"]))
    pool.conv.t.view(torch.bfloat16).copy_(gen.normal(slots * LAYERS * 3 * CONV))
    for kv in kvs:  # the slots hold a prompt already
        kv.advance(1000)
    kv = verify.KdaVerify(pool, [gen.weights() for _ in range(LAYERS)], total, slots)
    kv.v.p.t.view(torch.bfloat16).copy_(gen.normal(LAYERS * total * P_COLS))
    gates, out = gen.normal(LAYERS * total * 2 * WIDTH), torch.zeros(LAYERS * total * WIDTH, dtype=torch.bfloat16, device="cuda")
    gb, ob = _bytes(gates), _bytes(out)
    views = [(K.RowView.new(gb, j * total * 2 * WIDTH, 2 * WIDTH), K.RowView.new(gb, j * total * 2 * WIDTH + WIDTH, 2 * WIDTH),
              K.RowView.new(ob, j * total * WIDTH, WIDTH)) for j in range(LAYERS)]
    return {"pool": pool, "kvs": kvs, "round": kv, "windows": list(zip(kvs, rows)), "keep": keep, "views": views, "out": out}


def _run_verify_layer(case, s):
    form = K.Form.CHUNKED if case["form"] == "chunked" else K.Form.EXACT
    K.set_verify_form(form)
    K.set_commit_form(form)
    s["round"].verify(s["windows"])
    for j, (a, g, out) in enumerate(s["views"]):
        s["round"].layer(j, a, g, out)
    s["round"].commit(s["kvs"], s["keep"])
    pool = s["pool"]
    return s["out"], pool.state.t.view(torch.bfloat16 if case["state"] == "bf16" else torch.float32), pool.conv.t.view(torch.bfloat16)


def _prepare_verify_core(case, gen):
    rows, keep = _windows(case)
    total, slots = sum(rows), case["slots"]
    n = total * WIDTH
    s = {"rows": total, "layers": [gen.tokens(total) for _ in range(LAYERS)], "cu": _cu(rows), "off": _offsets(slots, STATE),
         "keep": torch.tensor(keep, dtype=torch.int32, device="cuda"), "state": gen.states(LAYERS * slots * STATE, "bf16")}
    s["states"] = list(s["state"].view(LAYERS, -1))
    s["out"] = torch.zeros(LAYERS, n, dtype=torch.bfloat16, device="cuda")
    s["outs"] = list(s["out"])
    s["saves"] = (torch.zeros(LAYERS, n, device="cuda"), torch.zeros(LAYERS, n, dtype=torch.bfloat16, device="cuda"),
                  torch.zeros(LAYERS, n, device="cuda"), torch.zeros(LAYERS, total * HEADS, device="cuda"))
    s["layer_saves"] = list(zip(*s["saves"]))
    return s


def _run_verify_core(case, s):
    chunked = case["form"] == "chunked"
    K.set_commit_form(K.Form.CHUNKED if chunked else K.Form.EXACT)
    for (q, k, v, g, beta), state, out, saves in zip(s["layers"], s["states"], s["outs"], s["layer_saves"]):
        core.decode_batch(HEADS, s["rows"], s["cu"], q, k, v, g, beta, state, s["off"], state_out=None, flags=core.TENSOR if chunked else 0,
                          out=out, saves=saves)
    core.commit_batch(HEADS, LAYERS, s["cu"], s["keep"], s["state"], case["slots"] * STATE, s["off"], s["saves"], s["rows"] * WIDTH, s["rows"] * HEADS)
    return s["out"], s["state"], s["saves"]


def _prepare_prefill_layer(case, gen):
    lanes, total = case["lanes"], case["lanes"] * case["rows"]
    s = {"stream": K.Stream(), "weights": gen.weights(), "p": gen.normal(total * P_COLS), "gates": gen.normal(total * 2 * WIDTH),
         "conv": gen.normal(lanes * 3 * CONV), "state": gen.states(lanes * STATE, case["state"]),
         "out": torch.zeros(total * WIDTH, dtype=torch.bfloat16, device="cuda"), "meta": K.BatchMeta.new(lanes)}
    s["meta"].set([K.Request(case["rows"], i * 3 * CONV, i * STATE) for i in range(lanes)])
    gates = _bytes(s["gates"])
    s["call"] = K.PrefillBatch(s["weights"], K.RowView.dense(_bytes(s["p"]), P_COLS), CONV, K.RowView.new(gates, 0, 2 * WIDTH),
                               K.RowView.new(gates, WIDTH, 2 * WIDTH), _bytes(s["conv"]), _bytes(s["state"]), K.StateOut.InPlace,
                               K.RowView.dense(_bytes(s["out"]), WIDTH), 0, K.PrefillWorkspace.new(HEADS, lanes, case["pass_rows"]))
    return s


def _run_prefill_layer(case, s):
    K.set_prefill_form(K.Form.CHUNKED if case["form"] == "chunked" else K.Form.EXACT)
    if case["state"] == "bf16":
        s["call"].launch_bf16_state(s["meta"], s["stream"])
    else:
        s["call"].launch(s["meta"], s["stream"])
    return s["out"], s["state"], s["conv"]


def _prepare_prefill_core(case, gen):
    heads, lengths, per = case["heads"], _lengths(case), case["heads"] * DK * DK
    rows, fused = case["rows"], case["fused"]
    s = {"tokens": gen.tokens(rows, heads), "cu": _cu(lengths), "max": max(lengths), "off": _offsets(len(lengths), per)}
    s["state"] = gen.states(len(lengths) * per, case["state"])
    s["state"].view(len(lengths), -1)[0::2] = 0  # every other sequence starts afresh
    s["gate"] = gen.normal(rows * heads * DK) if fused else None
    s["norm_w"] = gen.normal(DK, 0.1, mean=1.0) if fused else None
    s["out"] = torch.zeros(rows * heads * DK, dtype=torch.bfloat16, device="cuda")
    n = core.prefill_workspace_bytes(heads, len(lengths), case["chunks"]) if case["chunks"] else 0
    s["workspace"] = torch.empty(n, dtype=torch.uint8, device="cuda") if n else None
    return s


def _run_prefill_core(case, s):
    q, k, v, g, beta = s["tokens"]
    core.prefill_varlen(case["heads"], case["rows"], s["cu"], s["max"], q, k, v, g, beta, s["state"], s["off"], gate=s["gate"],
                        norm_w=s["norm_w"], out=s["out"], workspace=s["workspace"])
    return s["out"], s["state"]


def _prepare_proj(case, gen):
    rows = case["rows"]
    mat = lambda *shape: proj.Bf16Mat.dense(gen.normal(math.prod(shape), 0.02).view(*shape))
    empty = lambda n: torch.zeros(rows, n, dtype=torch.bfloat16, device="cuda")
    return {"w": proj.KdaProjW(mat(P_COLS, proj.HIDDEN), mat(2 * DK, proj.HIDDEN), mat(2, WIDTH, DK)), "o_proj": mat(proj.HIDDEN, WIDTH),
            "normed": gen.normal(rows * proj.HIDDEN).view(rows, -1), "core": gen.normal(rows * WIDTH).view(rows, -1),
            "p": empty(P_COLS), "fga": empty(2 * DK), "ag": empty(2 * WIDTH), "out": empty(proj.HIDDEN)}


def _run_proj(case, s):
    proj.kda_input_projections(s["normed"], case["rows"], s["w"], s["p"], s["fga"], s["ag"])
    proj.bf16(s["core"], WIDTH, 0, s["o_proj"], case["rows"], s["out"], proj.HIDDEN, 0)
    return s["p"], s["fga"], s["ag"], s["out"]


def _prepare_mark(case, gen):
    l, slots = _layout(case), case["slots"]
    pool = marks.KvPool(marks.KvConfig(l, 2 * slots, slots * l.mark_pages() + 7))
    kvs = [pool.slot() for _ in range(2 * slots)]
    pool.state.t.view(torch.bfloat16 if case["state"] == "bf16" else torch.float32).copy_(gen.states(2 * slots * LAYERS * STATE, case["state"]))
    pool.conv.t.view(torch.bfloat16).copy_(gen.normal(2 * slots * LAYERS * 3 * CONV))
    pool.tails.t.copy_(torch.randint(0, 256, (pool.tails.bytes(),), dtype=torch.uint8, device="cuda", generator=gen.g))
    for kv in kvs:
        kv.advance(4096)
    return {"pool": pool, "pairs": list(zip(kvs[:slots], kvs[slots:]))}


def _run_mark(case, s):
    held = []
    for source, fork in s["pairs"]:
        held.append(source.mark())
        fork.fork(source, source.tokens(), held[-1])
    for m in held:
        m.drop()
    pool = s["pool"]
    return pool.pages.t, pool.state.t, pool.conv.t, pool.tails.t


def prepare(case, seed):
    return {"case": case, **globals()["_prepare_" + case["kind"]](case, _Gen(seed))}


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state["case"], state)
