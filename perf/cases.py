"""What a program built on this library asks of it, as cases that can be timed.

The library is the attention half of a DiT block behind a C ABI.  A host program
opens a chain (h3_gpu_begin), enqueues the calls of one or more layers and submits;
one pass of a case is one such chain, begin to submit.  The families:

  layer   the attention half of the block from hidden state to hidden state, every
          layer with weights of its own: AdaLN norm, q/k/v projection, QK-norm +
          RoPE, block-causal attention, output projection, gated residual.
          calls = "fused": the recommended calls (projection with the norm and the
          rotation in its epilogue, bounded attention); "reference": the calls an
          unchanged host makes (two head norms, the rotation, the prefix attention).
  qkv     the same path from given q, k, v: fused QK-norm + RoPE, then block-causal
          attention, one output per layer; with several GPUs the heads are a rank's
          share.
  target  a later step of the edit path: only the target image's rows are new, the
          rest of every layer's K and V lies in a cache that the layer updates.
  text    token-causal attention of a text prefix or text tower (grouped heads), by
          one of the two causal entry points or by the prefix kernel.
  full    attention without a mask, one of the three entry points.

graph = True: the chain is one replay of a captured graph, as a host does that runs
the same layers for many steps.  Sizes are the benchmark's workloads, the shapes of
the SDPA benchmark and of the known-answer test, and what lies between them.
"""
import functools
import math

import numpy as np
import torch

from qwen_metal_b200 import abi

D = 128
SCALE = 1.0 / math.sqrt(D)
EPS = 1e-6
MODULATION_SLOTS, SCALE_SLOT, GATE_SLOT = 4, 0, 1


def listed():
    return [
        # The known-answer layout of the prefix kernel: one call, four runs, 149 rows.
        # The smallest thing a host asks for: launch and submit latency.
        _case("prefix-149", "text", entry="prefix", rows=149, heads=32, kv_heads=32),
        # A prompt through the text tower's attention: 32 query heads on 8 kv heads,
        # as many layers in a chain as a host flushes at a time.
        _case("text-gqa-412", "text", entry="causal", rows=412, heads=32, kv_heads=8, layers=6),
        # A 256^2 preview: 64 text rows and a 16x16 latent grid, a few layers per chain.
        _case("layer-256", "layer", text=64, gh=16, gw=16, heads=24, layers=4),
        # 512^2 turbo: few steps of the same layers, so the host replays a graph.
        _case("layer-512-graph", "layer", text=128, gh=32, gw=32, heads=24, layers=4, graph=True),
        # 1024^2 with classifier-free guidance: both branches as one batch, text padded
        # to a common length.
        _case("layer-1024-guided", "layer", batch=2, text=256, text_len0=200, text_len1=32, gh=64,
              gw=64, heads=24, layers=2),
        # The same shape from given q, k, v.
        _case("qkv-1024-guided", "qkv", batch=2, text=256, text_len0=200, text_len1=32, gh=64, gw=64,
              heads=24, layers=4),
        # 2048^2 with guidance: the largest image.
        _case("qkv-2048-guided", "qkv", batch=2, text=512, text_len0=512, text_len1=512, gh=128,
              gw=128, heads=24, layers=1),
        # One of eight GPUs at 1024^2: one guidance branch, six of the heads, replayed.
        _case("qkv-1024-share-graph", "qkv", text=256, text_len0=200, gh=64, gw=64, heads=6, layers=8,
              graph=True),
        # The first edit step by an unchanged host's calls: text, condition, target.
        _case("layer-edit-reference", "layer", calls="reference", text=256, ch=64, cw=64, gh=64,
              gw=64, heads=24, layers=1),
        # An odd prompt before a 768^2 image at the model's own width, unchanged host.
        _case("layer-768-reference", "layer", calls="reference", text=47, gh=48, gw=48, heads=32,
              layers=2),
        # A later edit step: 4096 target rows against 8448 cached ones.
        _case("target-1024", "target", text=256, ch=64, cw=64, gh=64, gw=64, heads=24, layers=2),
        # Image rows against all keys, ragged both ways (8188 queries, 8211 keys).
        _case("full-8188", "full", entry="flash", rows=8188, kv_rows=8211, heads=32),
    ]


def _case(name, family, **given):
    base = {
        "layer": dict(calls="fused", batch=1, text=0, text_len0=0, text_len1=0, ch=0, cw=0, gh=0, gw=0,
                      heads=24, layers=1, graph=False),
        "qkv": dict(batch=1, text=0, text_len0=0, text_len1=0, ch=0, cw=0, gh=0, gw=0, heads=24,
                    layers=1, graph=False),
        "target": dict(text=0, ch=0, cw=0, gh=0, gw=0, heads=24, layers=1, graph=False),
        "text": dict(entry="causal", rows=0, heads=32, kv_heads=8, layers=1, graph=False),
        "full": dict(entry="flash", rows=0, kv_rows=0, heads=32, layers=1, graph=False),
    }[family]
    case = dict(base, **given, family=family)
    if name:
        case["name"] = name
    return case


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        case = _draw(rng)
        if _cost(case) <= most:
            return case


def _spread(rng, lo, hi):
    """A whole number, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw(rng):
    family = rng.choice(["layer", "layer", "layer", "qkv", "qkv", "target", "text", "full"])
    graph = rng.random() < 0.3
    layers = rng.choice([1, 2, 3, 4])
    if family == "text":
        entry = rng.choice(["causal", "causal-prescaled", "prefix"])
        heads, kv_heads = rng.choice([(32, 8), (32, 32), (24, 24), (16, 8)])
        return _case("", family, entry=entry, rows=_spread(rng, 20, 2048), heads=heads,
                     kv_heads=kv_heads, layers=rng.choice([1, 2, 6]), graph=graph)
    if family == "full":
        rows = _spread(rng, 200, 16418)
        entry = rng.choice(["flash", "rect", "head-major"])
        kv_rows = rows if entry == "head-major" else rows + rng.choice([0, 0, rng.randint(1, 512)])
        return _case("", family, entry=entry, rows=rows, kv_rows=kv_rows,
                     heads=rng.choice([8, 24, 32]), graph=graph)
    gh, gw = _spread(rng, 12, 128), 0
    gw = max(10, min(128, int(round(gh * rng.choice([0.56, 0.75, 1.0, 1.0, 1.33, 1.78])))))
    text = _spread(rng, 9, 512)
    heads = rng.choice([3, 6, 12, 24, 24, 32] if family == "qkv" else [24, 24, 32])
    if family == "target":
        return _case("", family, text=text, ch=gh, cw=gw, gh=gh, gw=gw, heads=heads, layers=layers,
                     graph=graph)
    edit = rng.random() < 0.25
    condition = dict(ch=gh, cw=gw) if edit else {}
    guided = dict(batch=2, text_len0=rng.randint(1, text), text_len1=rng.randint(1, text))
    if family == "layer":
        calls = rng.choice(["fused", "fused", "reference"])
        if edit or calls == "reference" or rng.random() < 0.5:
            guided = {}
        return _case("", family, calls=calls, text=text, gh=gh, gw=gw, heads=heads, layers=layers,
                     graph=graph, **condition, **guided)
    if edit or rng.random() < 0.5:
        guided = {}
    return _case("", family, text=text, gh=gh, gw=gw, heads=heads, layers=layers, graph=graph,
                 **condition, **guided)


# ---- what a pass cannot do without ------------------------------------------


def _runs(c):
    runs = [(c["text"], 0)] if c["text"] else []
    if c["ch"]:
        runs.append((c["ch"] * c["cw"], 1))
    return runs + [(c["gh"] * c["gw"], 1)]


def _rows(c):
    return sum(n for n, _ in _runs(c)) if "gh" in c else c["rows"]


def _text_len(c):
    if not c.get("text_len0"):
        return None
    return np.array([c["text_len0"], c["text_len1"]][:c["batch"]], dtype=np.uint32)


def _visible(c):
    """Visible (query row, key) pairs of one head, over all batch items."""
    rows = _rows(c)
    if c["family"] == "target":
        return c["gh"] * c["gw"] * rows
    if c["family"] == "full":
        return rows * c["kv_rows"]
    if c["family"] == "text":
        return int(_text_limits(c).sum())
    limits, total, start = np.zeros(rows, np.int64), 0, 0
    for n, image in _runs(c):
        limits[start:start + n] = start + n if image else np.arange(start + 1, start + n + 1)
        start += n
    lens = _text_len(c)
    for b in range(c["batch"]):
        seen = limits
        if lens is not None:
            length, pad = int(lens[b]), c["text"]
            seen = limits - (np.minimum(pad, limits) - np.minimum(length, limits))
            seen[length:pad] = 0
        total += int(seen.sum())
    return total


def _text_limits(c):
    """Token-causal; the prefix entry point sees an interleaved prompt instead (text
    and image runs in turn, as the known-answer test lays them out)."""
    rows = c["rows"]
    limits = np.arange(1, rows + 1, dtype=np.uint32)
    if c["entry"] == "prefix":
        a, b = rows * 20 // 149, rows * 68 // 149
        limits[a:b] = b
        limits[rows * 85 // 149:] = rows
    return limits


def work(case):
    """Bytes and operations of one pass, call by call: what every call has to read and
    write once, and 2 operations per multiply-add of the visible scores, of P V and of
    the projections."""
    c, rows = case, _rows(case)
    heads, layers = c["heads"], c["layers"]
    attention = 4.0 * D * heads * _visible(c)
    if c["family"] == "text":
        sizes = rows * D * 2 * (2 * heads + 2 * c["kv_heads"])
        return {"bytes": float(layers * sizes), "flops": layers * attention}
    if c["family"] == "full":
        sizes = D * 2 * heads * 2 * (rows + c["kv_rows"])
        return {"bytes": float(layers * sizes), "flops": layers * attention}
    width = heads * D
    tables = 2 * rows * 64 * 4
    if c["family"] == "qkv":
        act = c["batch"] * rows * width * 2
        return {"bytes": float(layers * (4 * act + tables + 4 * act)), "flops": layers * attention}
    new = c["gh"] * c["gw"] if c["family"] == "target" else c["batch"] * rows
    act, weights = new * width * 2, width * width * 2
    projections = 2.0 * new * width * width * 4
    moved = 2 * act                       # AdaLN norm
    moved += act + 3 * weights + 3 * act  # q, k, v
    moved += 2 * act + weights            # output projection
    moved += 3 * act                      # gate
    if c["family"] == "target":
        moved += 6 * act + tables * new // rows                # q, k, v into place
        moved += 2 * act + 2 * rows * width * 2                # attention against the cache
    else:
        moved += 4 * act                                       # attention
        moved += tables + (4 * act if c["calls"] == "reference" else 0)  # norm + rotation
    return {"bytes": float(layers * moved), "flops": layers * (projections + attention)}


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def tolerance(case):
    # bf16 tensors between the stages and at the end, fp32 accumulation inside: about
    # one rounding (2^-9 of the value) per stage, 2e-3 to 5e-3 in the norm; a single
    # element is off by a few roundings of the row's values.
    return {"rel": 1e-2, "max": 0.1}


# ---- inputs -------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _gpu():
    """The program's one context."""
    return abi.Gpu()


class _Tensor:
    """A tensor of the library, freed with its last user (a view of it included)."""

    def __init__(self, handle, elements, typestr):
        gpu = _gpu()
        self.handle = handle
        self.__cuda_array_interface__ = {
            "shape": (elements,), "typestr": typestr, "version": 3, "strides": None,
            "data": (gpu.lib.qw_gpu_tensor_device_ptr(handle), False)}

    def __del__(self):
        gpu = _gpu()
        if gpu.handle:
            gpu.free(self.handle)

    def view(self, *shape):
        t = torch.as_tensor(self, device="cuda")
        return (t.view(torch.bfloat16) if t.dtype == torch.int16 else t).view(*shape)


class _State:
    """Inputs, weights and work buffers, the bound calls of a pass and its outputs."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.kept, self.calls, self.outputs, self.graph = [], [], [], None

    def __del__(self):
        if self.graph:
            _gpu().lib.qw_gpu_graph_free(self.graph)

    def new(self, *shape):
        n = int(np.prod(shape))
        t = _Tensor(_gpu().new_bf16(n), n, "<i2")
        self.kept.append(t)
        return t

    def normal(self, *shape, mean=0.0, std=1.0):
        t = self.new(*shape)
        torch.cuda.synchronize()  # the library clears a new tensor on its own stream
        t.view(*shape).normal_(mean, std, generator=self.gen)
        return t

    def f32(self, array):
        t = _Tensor(_gpu().f32(array), array.size, "<f4")
        self.kept.append(t)
        return t

    def u32(self, array):
        t = _Tensor(_gpu().u32(array), array.size, "<i4")
        self.kept.append(t)
        return t

    def call(self, name, *arguments):
        """Bind one call of the C ABI, its arguments converted once as a C host has them."""
        fn = getattr(_gpu().lib, name)
        bound = [_gpu().handle, *arguments]
        bound = [a.handle if isinstance(a, _Tensor) else a for a in bound]
        bound = [a if a is None or isinstance(a, kind) else kind(a)
                 for kind, a in zip(fn.argtypes, bound)]
        self.calls.append(functools.partial(fn, *bound))

    def output(self, tensor, *shape):
        self.outputs.append(tensor.view(*shape))


def prepare(case, seed):
    s = _State(seed)
    {"layer": _prepare_layer, "qkv": _prepare_qkv, "target": _prepare_target, "text": _prepare_text,
     "full": _prepare_full}[case["family"]](s, case)
    torch.cuda.synchronize()  # the inputs were made on torch's stream, the library has its own
    if case["graph"]:
        lib, handle = _gpu().lib, _gpu().handle
        _chain(s.calls)
        _gpu().begin()
        _gpu().check(lib.qw_gpu_graph_begin(handle), "graph begin")
        for call in s.calls:
            _gpu().check(call(), "capture")
        s.graph = lib.qw_gpu_graph_end(handle)
        _gpu().check(s.graph, "graph end")
        _gpu().submit()
        s.calls = []
        s.call("qw_gpu_graph_launch", s.graph)
    return s


def _layout(s, c):
    """Key limits, rotation tables and the row map of a joint token layout."""
    runs = _runs(c)
    limits = abi.prefix_limits(runs)
    grids = ([(c["ch"], c["cw"])] if c["ch"] else []) + [(c["gh"], c["gw"])]
    cos, sin = abi.rope_tables_blocks([g[0] for g in grids], [g[1] for g in grids],
                                      [c["text"]] + [0] * (len(grids) - 1))
    row_map = np.concatenate([np.full(n, 0 if image else 1, np.uint32) for n, image in runs])
    return limits, cos, sin, row_map


class _Weights:
    """One layer's weights."""

    def __init__(self, s, width):
        std = 1.0 / math.sqrt(width)
        self.q, self.k, self.v, self.out = (s.normal(width, width, std=std) for _ in range(4))
        self.norm_q, self.norm_k = (s.normal(D, mean=1.0, std=0.1) for _ in range(2))
        self.modulation = s.normal(2, MODULATION_SLOTS, width, std=0.3)


def _prepare_layer(s, c):
    rows, batch, heads = _rows(c), c["batch"], c["heads"]
    limits, cos, sin, row_map = _layout(s, c)
    width, new = heads * D, batch * rows
    lens = _text_len(c)
    s.lens = lens
    lens_at, pad = (abi._ptr(lens), c["text"]) if lens is not None else (None, 0)
    limits, cos, sin = s.u32(limits), s.f32(cos), s.f32(sin)
    row_map = s.u32(np.tile(row_map, batch))
    given = s.normal(new, width)
    hidden, normed, q, k, v, attn, proj = (s.new(new, width) for _ in range(7))
    bound = s.f32(np.zeros(2, np.float32))
    source = given
    for _ in range(c["layers"]):
        w = _Weights(s, width)
        s.call("qw_gpu_layer_norm_mod_bf16", normed, source, w.modulation, row_map, new, width,
               MODULATION_SLOTS, SCALE_SLOT, EPS)
        if c["calls"] == "fused":
            s.call("qw_gpu_qkv_norm_rope_bf16", q, k, v, normed, w.q, w.k, w.v, w.norm_q, w.norm_k,
                   cos, sin, bound, batch, rows, width, EPS)
            s.call("qw_gpu_attn_block_causal_bounded_bf16", attn, q, k, v, limits, bound, batch, rows,
                   heads, heads, D, lens_at, pad, SCALE)
        else:
            s.call("qw_gpu_qkv_bf16", q, k, v, normed, w.q, w.k, w.v, rows, width)
            s.call("h3_gpu_head_rms_norm_bf16", q, w.norm_q, rows, heads, D, EPS)
            s.call("h3_gpu_head_rms_norm_bf16", k, w.norm_k, rows, heads, D, EPS)
            s.call("qw_gpu_qk_rope_bf16", q, k, q, k, cos, sin, rows, heads, D)
            s.call("qw_gpu_flash_sdpa_prefix_bf16", attn, q, k, v, limits, rows, rows, heads, heads, D,
                   SCALE)
        s.call("h3_gpu_linear_bf16", proj, attn, w.out, None, new, width, width)
        s.call("h3_gpu_gate_bf16", hidden, source, proj, w.modulation, row_map, new, width,
               MODULATION_SLOTS, GATE_SLOT)
        source = hidden
    # The hidden state, and what the last layer leaves for a K/V cache.
    s.output(hidden, new, width)
    for t in (k, v, attn):
        s.output(t, new, heads, D)


def _prepare_qkv(s, c):
    rows, batch, heads = _rows(c), c["batch"], c["heads"]
    limits, cos, sin, _ = _layout(s, c)
    shape = (batch, rows, heads, D)
    lens = _text_len(c)
    s.lens = lens
    lens_at, pad = (abi._ptr(lens), c["text"]) if lens is not None else (None, 0)
    limits, cos, sin = s.u32(limits), s.f32(cos), s.f32(sin)
    q_work, k_work = s.new(*shape), s.new(*shape)
    bound = s.f32(np.zeros(2, np.float32))
    for _ in range(c["layers"]):
        q, k, v = (s.normal(*shape) for _ in range(3))
        norm_q, norm_k = (s.normal(D, mean=1.0, std=0.1) for _ in range(2))
        out = s.new(*shape)
        s.call("qw_gpu_qk_norm_rope_bound_bf16", q_work, k_work, q, k, norm_q, norm_k, cos, sin, bound,
               batch, rows, heads, D, EPS)
        s.call("qw_gpu_attn_block_causal_bounded_bf16", out, q_work, k_work, v, limits, bound, batch,
               rows, heads, heads, D, lens_at, pad, SCALE)
        s.output(out, *shape)
    s.output(q_work, *shape)
    s.output(k_work, *shape)


def _prepare_target(s, c):
    rows, heads, new = _rows(c), c["heads"], c["gh"] * c["gw"]
    width, base = heads * D, rows - new
    _, cos, sin, row_map = _layout(s, c)
    cos, sin, row_map = s.f32(cos[base:]), s.f32(sin[base:]), s.u32(row_map[base:])
    given = s.normal(new, width)
    hidden, normed, q, k, v, attn, proj = (s.new(new, width) for _ in range(7))
    source, caches = given, []
    for _ in range(c["layers"]):
        w = _Weights(s, width)
        k_cache, v_cache = s.normal(rows, width), s.normal(rows, width)
        s.call("qw_gpu_layer_norm_mod_bf16", normed, source, w.modulation, row_map, new, width,
               MODULATION_SLOTS, SCALE_SLOT, EPS)
        s.call("qw_gpu_qkv_bf16", q, k, v, normed, w.q, w.k, w.v, new, width)
        s.call("qw_gpu_qk_norm_rope_cache_bf16", q, k_cache, v_cache, k, v, w.norm_q, w.norm_k, cos,
               sin, rows, base, new, heads, D, EPS)
        s.call("qw_gpu_sdpa_rect_bf16", attn, q, k_cache, v_cache, new, rows, heads, D, SCALE)
        s.call("h3_gpu_linear_bf16", proj, attn, w.out, None, new, width, width)
        s.call("h3_gpu_gate_bf16", hidden, source, proj, w.modulation, row_map, new, width,
               MODULATION_SLOTS, GATE_SLOT)
        source = hidden
        caches += [k_cache, v_cache]
    s.output(hidden, new, width)
    for t in caches:
        s.output(t, rows, heads, D)


def _prepare_text(s, c):
    rows, heads, kv_heads = c["rows"], c["heads"], c["kv_heads"]
    limits = s.u32(_text_limits(c)) if c["entry"] == "prefix" else None
    for _ in range(c["layers"]):
        q, out = s.normal(rows, heads, D), s.new(rows, heads, D)
        k, v = s.normal(rows, kv_heads, D), s.normal(rows, kv_heads, D)
        if c["entry"] == "prefix":
            s.call("qw_gpu_flash_sdpa_prefix_bf16", out, q, k, v, limits, rows, rows, heads, kv_heads, D,
                   SCALE)
        else:
            name = "qw_gpu_gqa_causal_bf16" if c["entry"] == "causal" else "h3_gpu_gqa_causal_bf16"
            s.call(name, out, q, k, v, rows, heads, kv_heads, D, SCALE)
        s.output(out, rows, heads, D)


def _prepare_full(s, c):
    rows, kv_rows, heads = c["rows"], c["kv_rows"], c["heads"]
    q, out = s.normal(rows, heads, D), s.new(rows, heads, D)
    k, v = s.normal(kv_rows, heads, D), s.normal(kv_rows, heads, D)
    if c["entry"] == "head-major":
        s.call("h3_gpu_sdpa_bf16_head_major_output", out, q, k, v, rows, heads, D, SCALE)
        s.output(out, heads, rows, D)
    else:
        name = "qw_gpu_flash_sdpa_bf16" if c["entry"] == "flash" else "qw_gpu_sdpa_rect_bf16"
        s.call(name, out, q, k, v, rows, kv_rows, heads, D, SCALE)
        s.output(out, rows, heads, D)


# ---- a pass ---------------------------------------------------------------------


def _chain(calls):
    gpu = _gpu()
    gpu.begin()
    for call in calls:
        if not call():
            gpu.check(0, "enqueue")
    gpu.submit()


def run(state):
    _chain(state.calls)
    return state.outputs
