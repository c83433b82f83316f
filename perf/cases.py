"""Workloads of the attention + KV-cache path, for timing and for comparing two builds.

Each case is one call sequence that a program on top of this library makes, over the geometries of
the benchmark's configurations (hydra_b200/workloads.py): GPT-OSS (64 query / 8 KV heads, d 64,
window 128 or full, sinks), Gemma (16/8, d 256, window 1024 or full, q/k/v norms, scale 1; its wide
global layers are 16/2, d 512) and Qwen (16/2, d 256, 64 rotated dims, q/k norms, interleaved output
gate).  Kinds:

  decode   a generated token of one sequence: `layer_step` with one token, per layer
  batch    a decode step of many sequences: `write_key_value_batch`, then `attention`, per layer
  prefill  a prompt (or the rest of one, when `position` > 0): `prefill_chunks` per layer; with
           `then_decode` the first generated token's `layer_step` follows
  host     a prompt whose activations live in pinned host memory: `prefill_host`
  project  the projections around attention: `rms_norm`, `linear_group` (q, k, v), `linear` (o)
  forward  `AttentionStackRunner.verify`: hidden states in host memory through a stack of layers

Activations are N(0, 1) as the projections of normalised hidden states are, weights N(0, 0.02),
norm weights near 1, cached rows N(0, 1).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import hydra_b200 as hb
from hydra_b200 import capi
from hydra_b200.runner import AttentionLayerWeights, AttentionStackRunner

# name: (q_heads, kv_heads, head_dim, window, theta, rotated pairs or None, q/k norm, v norm, sinks, gate)
GEOMETRIES = {
    "gpt-oss-window": (64, 8, 64, 128, 150000.0, None, False, False, True, False),
    "gpt-oss-full": (64, 8, 64, 0, 150000.0, None, False, False, True, False),
    "gemma-local": (16, 8, 256, 1024, 1e4, None, True, True, False, False),
    "gemma-global": (16, 8, 256, 0, 1e6, None, True, True, False, False),
    "gemma-global-wide": (16, 2, 512, 0, 1e6, 64, True, True, False, False),
    "qwen": (16, 2, 256, 0, 1e7, 32, True, False, False, True),
}
# Projections: name: (hidden, q_proj rows, k and v rows, o_proj columns, bias)
PROJECTIONS = {
    "gpt-oss": (2880, 4096, 512, 4096, True),
    "gemma": (2816, 4096, 2048, 4096, False),
    "qwen": (2048, 8192, 512, 4096, False),
}
GEMMA_STACK = "gemma-local*5+gemma-global"
GPT_OSS_PAIR = "gpt-oss-window+gpt-oss-full"


def listed():
    return [
        # A generated token in a windowed GPT-OSS layer: the smallest call, all latency.
        dict(name="decode_window128", kind="decode", layers="gpt-oss-window", position=511, io="bf16"),
        # The same token in a full-attention layer after a 4096-token prompt.
        dict(name="decode_full_4096", kind="decode", layers="gpt-oss-full", position=4095, io="bf16"),
        # A long conversation on a gated layer with two KV heads.
        dict(name="decode_gated_32768", kind="decode", layers="qwen", position=32767, io="bf16"),
        # A serving step: 64 sequences of ragged lengths, one windowed and one full layer.
        dict(name="batch_64_ragged", kind="batch", layers=GPT_OSS_PAIR, sequences=64, longest=16384, paged=False, io="bf16"),
        # A short prompt in small chunks on a windowed layer.
        dict(name="prefill_window128_512", kind="prefill", layers="gpt-oss-window", tokens=512, position=0, chunk=128,
             then_decode=False, io="bf16"),
        # The headline: a 4096-token prompt in 512-token chunks, full attention.
        dict(name="prefill_full_4096", kind="prefill", layers="gpt-oss-full", tokens=4096, position=0, chunk=512,
             then_decode=False, io="bf16"),
        # The largest: a long prompt through a Gemma stack, five local layers to one global.
        dict(name="prefill_stack_8192", kind="prefill", layers=GEMMA_STACK, tokens=8192, position=0, chunk=512,
             then_decode=False, io="bf16"),
        # A second turn of a conversation: an odd number of new tokens behind an odd history, fp32
        # activations as the reference's runners hold them.
        dict(name="prefill_gated_resume", kind="prefill", layers="qwen", tokens=777, position=1291, chunk=512,
             then_decode=False, io="f32"),
        # A turn on a wide Gemma layer: the prompt and the first token after it.
        dict(name="turn_wide_1000", kind="prefill", layers="gemma-global-wide", tokens=1000, position=0, chunk=512,
             then_decode=True, io="bf16"),
        # A layer's projections for a prompt.
        dict(name="project_4096", kind="project", model="gpt-oss", tokens=4096),
        # A generated token through the runner, hidden state in and out of host memory.
        dict(name="forward_token", kind="forward", tokens=1, position=2000),
        # The headline prompt with its activations in host memory.
        dict(name="host_prompt_4096", kind="host", layers="gpt-oss-full", tokens=4096, position=0, chunk=512, io="bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "batch", "prefill", "prefill", "prefill", "project", "forward", "host"])
    io = rng.choice(["bf16", "bf16", "f32"])
    if kind == "decode":
        layers = rng.choice(["gpt-oss-window", "gpt-oss-full", "gemma-local", "gemma-global", "gemma-global-wide", "qwen"])
        return dict(kind=kind, layers=layers, position=_log_int(rng, 60, 32767), io=io)
    if kind == "batch":
        return dict(kind=kind, layers=rng.choice([GPT_OSS_PAIR, "gpt-oss-full", "qwen"]), sequences=_log_int(rng, 2, 64),
                    longest=_log_int(rng, 512, 16384), paged=rng.random() < 0.4, io=io)
    if kind == "prefill":
        layers = rng.choice(["gpt-oss-window", "gpt-oss-full", GEMMA_STACK, "gemma-local", "gemma-global", "qwen",
                             "gemma-global-wide"])
        most = 1000 if layers == "gemma-global-wide" else 8192
        tokens = _log_int(rng, 40, most)
        # A later turn stays below the context at which windowed layers become rings: a pass that is run
        # again finds its history where it was.
        behind = min(most, 8000) - tokens
        return dict(kind=kind, layers=layers, tokens=tokens,
                    position=rng.randint(1, behind) if behind > 0 and rng.random() < 0.5 else 0,
                    chunk=rng.choice([128, 256, 512]), then_decode=rng.random() < 0.3, io=io)
    if kind == "project":
        return dict(kind=kind, model=rng.choice(sorted(PROJECTIONS)), tokens=_log_int(rng, 1, 4096))
    if kind == "forward":
        return dict(kind=kind, tokens=_log_int(rng, 1, 256), position=_log_int(rng, 60, 3500))
    return dict(kind=kind, layers=rng.choice(["gpt-oss-window", "gpt-oss-full", "qwen"]), tokens=_log_int(rng, 200, 4096),
                position=0, chunk=rng.choice([128, 256, 512]), io="bf16")


# ---- helpers --------------------------------------------------------------------------------------

def _layers(text):
    """'a*5+b' -> [a, a, a, a, a, b]"""
    out = []
    for part in text.split("+"):
        name, _, times = part.partition("*")
        out += [name] * int(times or 1)
    return out


_shared = {}


def _context():
    # One context per process, as a program has one per device.
    if "context" not in _shared:
        _shared["context"] = hb.Context(0)
    return _shared["context"]


def _rope(name, positions):
    """A geometry's rotation table: built at load time from the configuration and kept."""
    _, _, d, _, theta, pairs, *_ = GEOMETRIES[name]
    key = (d, theta, pairs, positions)
    if key not in _shared:
        _shared[key] = hb.RopeTable(_context(), hb.inverse_frequencies(d, theta, pairs), positions)
    return _shared[key]


class _DeviceArray:
    """A device buffer of a cache, described for torch (bf16 bits as int16).  torch keeps this object for as long as
    the tensor, and so the cache with it."""

    def __init__(self, cache, pointer, shape):
        self.cache = cache
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<i2", data=(pointer, False), version=2)


def _planes(cache, index, name, sequences, paged):
    """A layer's key and value rows in the cache, [sequences][kv_heads][capacity][head_dim]."""
    info = cache.layer(index)
    _, kv, d, *_ = GEOMETRIES[name]
    in_pool = paged and info.ring_size == 0
    shape = (1 if in_pool else sequences, kv, info.capacity, d)
    return [torch.as_tensor(_DeviceArray(cache, p, shape), device="cuda").view(torch.bfloat16) for p in (info.keys, info.values)]


def _ragged(case):
    # Uniform in [longest / 16, longest], the same lengths whatever the seed of the values.
    return [int(n) for n in np.random.default_rng(7).integers(max(2, case["longest"] // 16), case["longest"] + 1, case["sequences"])]


class _State:
    pass


def prepare(case, seed):
    if case["kind"] == "project":
        return _prepare_project(case, seed)
    if case["kind"] == "forward":
        return _prepare_forward(case, seed)
    return _prepare_attention(case, seed)


# ---- attention over the cache -----------------------------------------------------------------------

def _prepare_attention(case, seed):
    s = _State()
    s.case, kind = case, case["kind"]
    s.names = _layers(case["layers"])
    s.backend = hb.AttentionBackend(_context())
    gen = torch.Generator(device="cuda").manual_seed(seed)
    bf = torch.bfloat16
    dtype, io = (bf, capi.HC_BF16) if case["io"] == "bf16" else (torch.float32, capi.HC_F32)

    def normal(*shape, dtype=dtype, std=1.0):
        return (torch.randn(shape, device="cuda", dtype=torch.float32, generator=gen) * std).to(dtype)

    s.sequences, paged, pages = 1, False, 0
    if kind == "decode":
        rows, history, longest, chunk = 1, [case["position"]], case["position"] + 1, 512
    elif kind == "batch":
        lengths = _ragged(case)
        s.sequences = rows = len(lengths)
        s.positions, s.ids = [n - 1 for n in lengths], list(range(rows))
        history, longest, chunk, paged = s.positions, case["longest"], 512, case["paged"]
        pages = sum((n + 127) // 128 for n in lengths) if paged else 0
    else:
        rows = case["tokens"] + (1 if case.get("then_decode") else 0)
        history, longest, chunk = [case["position"]], case["position"] + rows, case["chunk"]
    context = (longest + 255) // 128 * 128               # the program's limit: this pass and room for a reply

    descs = [dict(q_heads=g[0], kv_heads=g[1], head_dim=g[2], window=g[3]) for g in (GEOMETRIES[n] for n in s.names)]
    s.cache = hb.KVCache(_context(), descs, context, prefill_chunk=chunk, max_seqs=s.sequences, total_pages=pages)
    s.layers = []
    for index, name in enumerate(s.names):
        q_heads, kv, d, window, _, _, qk_norm, v_norm, sinks, gate = GEOMETRIES[name]
        layer = _State()
        layer.q = normal(rows, q_heads, d * (2 if gate else 1))
        layer.k, layer.v = normal(rows, kv, d), normal(rows, kv, d)
        layer.out = torch.zeros((rows, q_heads, d), device="cuda", dtype=dtype)
        if kind == "host":
            for field in ("q", "k", "v", "out"):
                device = getattr(layer, field)
                pinned = torch.empty(device.shape, dtype=device.dtype, pin_memory=True)
                pinned.copy_(device)
                setattr(layer, field, pinned)
        layer.params = hb.AttnParams(
            q_heads=q_heads, kv_heads=kv, head_dim=d, window=window,
            sm_scale=1.0 if name.startswith("gemma") else 1.0 / math.sqrt(d), io_dtype=io,
            sinks=normal(q_heads, dtype=bf) if sinks else None,
            norm_q=1 if qk_norm else 0, norm_k=1 if qk_norm else 0, norm_v=2 if v_norm else 0,
            q_norm_weight=1 + normal(d, dtype=bf, std=0.1) if qk_norm else None,
            k_norm_weight=1 + normal(d, dtype=bf, std=0.1) if qk_norm else None,
            rope=_rope(name, context), gate_layout=capi.HC_GATE_INTERLEAVED if gate else capi.HC_GATE_NONE)
        # Earlier turns: rows that were normalised and rotated when they came, stored as they are.
        plain = hb.AttnParams(q_heads=q_heads, kv_heads=kv, head_dim=d, window=window, io_dtype=capi.HC_BF16)
        ring = s.cache.layer(index).ring_size
        for seq, length in enumerate(history):
            first = max(0, length - window) // 128 * 128 if ring else 0        # a ring keeps its window only
            if length > first:
                k, v = normal(length - first, kv, d, dtype=bf), normal(length - first, kv, d, dtype=bf)
                step = 128 if ring else length
                for at in range(first, length, step):
                    s.backend.write_key_value(s.cache, index, k[at - first:], v[at - first:], min(step, length - at), at,
                                              plain, seq=seq)
        layer.rows = _planes(s.cache, index, name, s.sequences, paged)
        s.layers.append(layer)
    torch.cuda.synchronize()
    return s


def _run_attention(s):
    case, be, kind = s.case, s.backend, s.case["kind"]
    for index, layer in enumerate(s.layers):
        if kind == "decode":
            be.layer_step(s.cache, index, layer.q, layer.k, layer.v, layer.out, 1, case["position"], layer.params)
        elif kind == "batch":
            be.write_key_value_batch(s.cache, index, layer.k, layer.v, s.ids, s.positions, layer.params)
            be.attention(s.cache, index, layer.q, layer.out, s.positions, layer.params, seq_ids=s.ids)
        elif kind == "host":
            be.prefill_host(s.cache, index, layer.q, layer.k, layer.v, layer.out, case["tokens"], case["position"],
                            case["chunk"], layer.params)
        else:
            be.prefill_chunks(s.cache, index, layer.q, layer.k, layer.v, layer.out, case["tokens"], case["position"],
                              case["chunk"], layer.params)
            if case["then_decode"]:
                n = case["tokens"]
                be.layer_step(s.cache, index, layer.q[n:], layer.k[n:], layer.v[n:], layer.out[n:], 1, case["position"] + n,
                              layer.params)
    return {"out": [layer.out for layer in s.layers], "cache": [layer.rows for layer in s.layers]}


def _work_attention(case):
    if case["kind"] == "batch":
        spans = [(n - 1, n) for n in _ragged(case)]
    elif case["kind"] == "decode":
        spans = [(case["position"], case["position"] + 1)]
    else:
        spans = [(case["position"], case["position"] + case["tokens"] + (1 if case.get("then_decode") else 0))]
    io = 2 if case["io"] == "bf16" else 4
    nbytes = flops = 0.0
    for name in _layers(case["layers"]):
        q_heads, kv, d, window, _, _, _, _, _, gate = GEOMETRIES[name]
        for first, end in spans:
            p = np.arange(first, end, dtype=np.float64)
            visible = np.minimum(p + 1, window) if window else p + 1
            flops += 4.0 * d * q_heads * float(visible.sum())
            oldest = max(0, first - window + 1) if window else 0
            nbytes += (end - first) * d * io * (q_heads * (3 if gate else 2) + 2 * kv)     # q (and gate), out, k, v
            nbytes += (end - oldest) * kv * d * 2 * 2                                      # cached rows, read or written
    return {"bytes": nbytes, "flops": flops}


# ---- projections and the runner ----------------------------------------------------------------------

def _prepare_project(case, seed):
    s = _State()
    s.case = case
    s.backend = hb.AttentionBackend(_context())
    gen = torch.Generator(device="cuda").manual_seed(seed)
    hidden, q_rows, kv_rows, o_cols, bias = PROJECTIONS[case["model"]]
    n, bf = case["tokens"], torch.bfloat16

    def normal(*shape, std=1.0, dtype=bf):
        return (torch.randn(shape, device="cuda", dtype=torch.float32, generator=gen) * std).to(dtype)

    s.widths = [q_rows, kv_rows, kv_rows]
    s.hidden = normal(n, hidden, dtype=torch.float32)
    s.norm = 1 + normal(hidden, std=0.1)
    s.w = [normal(rows, hidden, std=0.02) for rows in s.widths]
    s.b = [normal(rows, std=0.02) if bias else None for rows in s.widths]
    s.wo, s.bo = normal(hidden, o_cols, std=0.02), normal(hidden, std=0.02) if bias else None
    s.attended = normal(n, o_cols)
    s.normed = torch.zeros((n, hidden), device="cuda", dtype=bf)
    s.y = [torch.zeros((n, rows), device="cuda", dtype=bf) for rows in s.widths]
    s.out = torch.zeros((n, hidden), device="cuda", dtype=torch.float32)
    return s


def _run_project(s):
    n, hidden = s.hidden.shape
    s.backend.rms_norm(s.hidden, s.norm, s.normed, n, hidden, 1e-5)
    s.backend.linear_group(s.normed, s.w, s.b, s.y, n, hidden)
    s.backend.linear(s.attended, s.wo, s.bo, s.out, n, s.attended.shape[1], hidden, residual=s.hidden)
    return {"normed": s.normed, "qkv": s.y, "out": s.out}


def _work_project(case):
    hidden, q_rows, kv_rows, o_cols, _ = PROJECTIONS[case["model"]]
    n, rows = case["tokens"], q_rows + 2 * kv_rows
    weights = 2.0 * hidden * (rows + o_cols)
    return {"bytes": weights + n * (4.0 * hidden + 2 * rows + 2 * o_cols + 4 * hidden), "flops": n * weights}


FORWARD_WINDOWS = (128, 0)          # the runner's two layers


def _prepare_forward(case, seed):
    s = _State()
    s.case = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    hidden, q_rows, kv_rows, _, _ = PROJECTIONS["gpt-oss"]
    q_heads, kv, d = GEOMETRIES["gpt-oss-full"][:3]

    def normal(*shape, std=1.0):
        return (torch.randn(shape, device="cuda", generator=gen) * std).cpu().numpy()

    weights = [AttentionLayerWeights(
        input_norm=1 + normal(hidden, std=0.1), wq=normal(q_rows, hidden, std=0.02), bq=normal(q_rows, std=0.02),
        wk=normal(kv_rows, hidden, std=0.02), bk=normal(kv_rows, std=0.02), wv=normal(kv_rows, hidden, std=0.02),
        bv=normal(kv_rows, std=0.02), wo=normal(hidden, q_rows, std=0.02), bo=normal(hidden, std=0.02),
        sinks=normal(q_heads), window=window, inv_freq=hb.inverse_frequencies(d, 150000.0))
        for window in FORWARD_WINDOWS]
    s.runner = AttentionStackRunner(_context(), weights, hidden, q_heads, kv, d, context_length=4096)
    position = case["position"]
    for index, window in enumerate(FORWARD_WINDOWS):
        plain = hb.AttnParams(q_heads=q_heads, kv_heads=kv, head_dim=d, window=window, io_dtype=capi.HC_BF16)
        k, v = (torch.randn((position, kv, d), device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2))
        s.runner.backend.write_key_value(s.runner.kv_cache, index, k, v, position, 0, plain)
    torch.cuda.synchronize()
    s.runner.kv_cache.advance(position)
    s.hidden = normal(case["tokens"], hidden)
    s.rows = [_planes(s.runner.kv_cache, i, "gpt-oss-full", 1, False) for i in range(len(FORWARD_WINDOWS))]
    return s


def _run_forward(s):
    if s.runner.position != s.case["position"]:
        s.runner.rewind(s.case["position"])              # the draft is turned down: back to where it began
    return {"hidden": s.runner.verify(s.hidden), "cache": s.rows}


def _work_forward(case):
    layers = {0: "gpt-oss-full", 128: "gpt-oss-window"}
    total = {"bytes": 0.0, "flops": 0.0}
    for window in FORWARD_WINDOWS:
        attention = _work_attention(dict(kind="prefill", layers=layers[window], tokens=case["tokens"], position=case["position"], io="bf16"))
        project = _work_project(dict(model="gpt-oss", tokens=case["tokens"]))
        for key in total:
            total[key] += attention[key] + project[key]
    return total


# ---- what is measured -----------------------------------------------------------------------------------

def run(state):
    kind = state.case["kind"]
    if kind == "project":
        return _run_project(state)
    if kind == "forward":
        return _run_forward(state)
    return _run_attention(state)


def work(case):
    if case["kind"] == "project":
        return _work_project(case)
    if case["kind"] == "forward":
        return _work_forward(case)
    return _work_attention(case)


def tolerance(case):
    # bf16 operands (queries, softmax weights, cached rows) with fp32 accumulation: a few units of
    # 2^-9 per element.  The projections' own sums are fp32, of bf16 operands that may round the other way.
    return {"rel": 5e-3, "max": 0.1} if case["kind"] == "project" else {"rel": 1e-2, "max": 0.1}
