"""The work a user of this framework has it do, as cases that can be timed and compared.

Two model shapes appear throughout: `dense` (32 query / 8 kv heads, head_dim 128, NeoX RoPE) and `hybrid` (24 query / 4 kv
heads, head_dim 256, sectioned RoPE, K norm, gated output).  A cache is `q8_0` (32 int8 + one fp16 scale), `row` (int8, one
scale per row) or `f16` (the storage class's default mode); activations are fp16 or fp32.

  step     one layer of a decode step, called eagerly: append a token, attend the whole context
  decode   a decode step over all attention layers, captured once in a CUDA graph and replayed (position on the device); the
           hybrid shape starts each layer with the query-side split/norm/RoPE
  batched  one decode attention launch per layer for many sessions of mixed length, split size planned on the host
  prefill  a chunk of new tokens over an existing prefix: per layer the store kernel, then the suffix attention
  append   the store kernel alone (filling a cache from K/V that exist already)
  reuse    the snapshot pool's round trip: capture a session's prefix, then restore it into another session's caches
"""
import math
import random

import torch

from miinfer_b200 import kv

SHAPES = {"dense": dict(hq=32, hkv=8, d=128, rope=kv.RopeMode.NEOX_FULL), "hybrid": dict(hq=24, hkv=4, d=256, rope=kv.RopeMode.SECTIONED64)}
THETA = 1.0e6


def listed():
    return [
        # the smallest call: one layer's decode step at a 4K context, where launch latency and host work are the time
        {"name": "step-dense-4k", "kind": "step", "shape": "dense", "cache": "q8_0", "act": "f16", "context": 4096},
        # the decode benchmark: a 36-layer step at a 32K context
        {"name": "decode-dense-32k", "kind": "decode", "shape": "dense", "cache": "q8_0", "act": "f16", "context": 32768, "layers": 36},
        # one very long session
        {"name": "decode-dense-128k", "kind": "decode", "shape": "dense", "cache": "q8_0", "act": "f16", "context": 131072, "layers": 16},
        # a chat in progress on the hybrid model, one scale per row and fp32 activations, an odd length
        {"name": "decode-hybrid-7777", "kind": "decode", "shape": "hybrid", "cache": "row", "act": "f32", "context": 7777, "layers": 16},
        # the same model with the cache left in its default fp16 mode
        {"name": "decode-hybrid-f16-6001", "kind": "decode", "shape": "hybrid", "cache": "f16", "act": "f16", "context": 6001, "layers": 16},
        # serving: 80 sessions of 512 to 16384 tokens
        {"name": "batched-dense-80", "kind": "batched", "shape": "dense", "cache": "q8_0", "act": "f16", "sessions": 80, "shortest": 512,
         "longest": 16384, "mix": 42, "layers": 4},
        # serving the hybrid model to a few dozen shorter sessions
        {"name": "batched-hybrid-24", "kind": "batched", "shape": "hybrid", "cache": "q8_0", "act": "f16", "sessions": 24, "shortest": 200,
         "longest": 6000, "mix": 7, "layers": 4},
        # the prefill benchmark: a 512-token chunk over an 8192-token prefix
        {"name": "prefill-hybrid-512-8192", "kind": "prefill", "shape": "hybrid", "cache": "q8_0", "act": "f16", "prefix": 8192, "tokens": 512,
         "layers": 16},
        # a fresh prompt: nothing before the chunk
        {"name": "prefill-dense-2048-0", "kind": "prefill", "shape": "dense", "cache": "q8_0", "act": "f16", "prefix": 0, "tokens": 2048, "layers": 8},
        # a short user turn after a reused prefix, fp32 activations, odd sizes
        {"name": "prefill-hybrid-37-3001", "kind": "prefill", "shape": "hybrid", "cache": "row", "act": "f32", "prefix": 3001, "tokens": 37,
         "layers": 16},
        # filling caches from an 8192-token chunk
        {"name": "append-dense-8192", "kind": "append", "shape": "dense", "cache": "q8_0", "act": "f16", "tokens": 8192, "layers": 12},
        # keeping a 4096-token prefix and handing it to another session
        {"name": "reuse-hybrid-4096", "kind": "reuse", "shape": "hybrid", "cache": "q8_0", "act": "f16", "prefix": 4096, "layers": 16},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    case = {"kind": rng.choice(["step", "decode", "decode", "batched", "prefill", "prefill", "append", "reuse"]),
            "shape": rng.choice(["dense", "hybrid"]), "cache": rng.choice(["q8_0", "q8_0", "row", "f16"]), "act": rng.choice(["f16", "f32"])}
    kind, position = case["kind"], _row_bytes(case) * 2 * SHAPES[case["shape"]]["hkv"]   # cache bytes of one position of a layer
    if kind == "step":
        case.update(context=_spread(rng, 128, 32768))
    elif kind == "decode":
        case.update(context=_spread(rng, 512, 131072))
        case.update(layers=max(1, min(36 if case["shape"] == "dense" else 16, int(2.5e9 / (case["context"] * position)))))
    elif kind == "batched":
        longest = _spread(rng, 1024, 16384)
        case.update(sessions=min(_spread(rng, 2, 96), int(4.0e9 / (longest * position))), shortest=_spread(rng, 128, longest), longest=longest,
                    mix=rng.randrange(1 << 20))
        case.update(layers=max(1, min(8, int(4.0e9 / (case["sessions"] * longest * position)))))
    elif kind == "prefill":
        case.update(prefix=rng.choice([0, _spread(rng, 256, 32768), _spread(rng, 256, 32768)]), tokens=_spread(rng, 16, 4096))
        while work(case)["flops"] > 1.5e12:
            case["tokens"] //= 2
        case.update(layers=max(1, min(16, int(1.5e12 / work(case)["flops"]))))
    elif kind == "append":
        case.update(tokens=_spread(rng, 16, 16384))
        case.update(layers=max(1, min(36, int(6.0e8 / (case["tokens"] * position)))))
    else:
        case.update(prefix=_spread(rng, 256, 8192), layers=rng.randint(4, 16))
    return case


def _lengths(case):
    """The sessions' lengths, uniform between the bounds; a fifth of the sessions share one restored prefix of a quarter of the longest."""
    rng, n = random.Random(case["mix"]), case["sessions"]
    shared = max(case["shortest"], case["longest"] // 4)
    return [rng.randint(case["shortest"], case["longest"]) if i < n - n // 5 else shared for i in range(n)]


def _row_bytes(case):
    """Bytes of one side (K or V) of one cache row."""
    d = SHAPES[case["shape"]]["d"]
    return {"q8_0": d + 2 * (d // 32), "row": d + 2, "f16": 2 * d}[case["cache"]]


def work(case):
    s, kind = SHAPES[case["shape"]], case["kind"]
    hq, hkv, d = s["hq"], s["hkv"], s["d"]
    act, row, layers = (2 if case["act"] == "f16" else 4), _row_bytes(case), case.get("layers", 1)
    if kind in ("step", "decode"):
        ctx = case["context"]
        gated = case["shape"] == "hybrid"
        query = hq * d * (act + 4 if gated else act)                  # q, and for the hybrid shape its fp32 gate
        if gated and kind == "decode":
            query = 2 * hq * d * act                                  # the projection's [q | gate]
        bytes_ = ctx * hkv * row * 2 + query + hq * d * 4 + 2 * hkv * d * act
        return {"bytes": layers * bytes_, "flops": layers * 4.0 * d * hq * ctx}
    if kind == "batched":
        total = sum(_lengths(case))
        return {"bytes": layers * (total * hkv * row * 2 + case["sessions"] * hq * d * (act + 4)), "flops": layers * 4.0 * d * hq * total}
    if kind == "prefill":
        p, t = case["prefix"], case["tokens"]
        gate = 4 if case["shape"] == "hybrid" else 0
        bytes_ = (p + t) * hkv * row * 2 + t * hkv * d * 2 * act + t * hq * d * (act + gate + 4)
        return {"bytes": layers * bytes_, "flops": layers * 4.0 * d * hq * (t * p + t * (t + 1) / 2)}
    if kind == "append":
        return {"bytes": layers * case["tokens"] * hkv * 2 * (d * act + row), "flops": 0}
    return {"bytes": layers * 4 * case["prefix"] * hkv * row * 2, "flops": 0}   # cache -> snapshot -> other cache


def tolerance(case):
    if case["kind"] in ("append", "reuse"):
        return "exact"
    if case["kind"] == "prefill":
        return {"rel": 1e-3}     # weights and dequantised rows enter the tensor cores as fp16 (2^-11 each)
    # int8 caches: the query is taken as 15-bit and the weights as 16-bit fixed point against exact int8 sums (oracle: 7e-5);
    # fp16 caches: fp32 sums
    return {"rel": 2e-5 if case["cache"] == "f16" else 2e-4}


class Caches:
    """All layers' planes of one session, side by side in one allocation per plane, and the layers' views."""

    def __init__(self, case, capacity, layers):
        s = SHAPES[case["shape"]]
        h, d, q8 = s["hkv"], s["d"], case["cache"] != "f16"
        qb = 32 if case["cache"] == "q8_0" else d
        data = lambda: torch.zeros(layers, h, capacity, d, dtype=torch.int8 if q8 else torch.float16, device="cuda")
        scales = lambda: torch.zeros(layers, h, capacity, d // qb, dtype=torch.float16, device="cuda") if q8 else None
        self.k, self.v, self.ks, self.vs = data(), data(), scales(), scales()
        ptr = lambda t, l: t[l].data_ptr() if t is not None else None
        mode = int(kv.KvCacheQuantMode.kQ8Q8 if q8 else kv.KvCacheQuantMode.kFp16Fp16)
        plain = lambda t, l, want: ptr(t, l) if want else None
        self.views = [kv.AttentionKvCacheView(plain(self.k, l, not q8), plain(self.v, l, not q8), plain(self.k, l, q8), ptr(self.ks, l),
                                              plain(self.v, l, q8), ptr(self.vs, l), capacity, h, d, qb, mode) for l in range(layers)]

    def planes(self):
        return [t for t in (self.k, self.v, self.ks, self.vs) if t is not None]


def _fill(case, views, tokens, g):
    """Existing context: N(0, 1) rows through the store kernel."""
    s = SHAPES[case["shape"]]
    width = s["hkv"] * s["d"]
    for view in views:
        for base in range(0, tokens, 8192):
            n = min(8192, tokens - base)
            k, v = (torch.randn(n, width, generator=g, device="cuda").half() for _ in range(2))
            kv.launch_kv_store_quant(view, k, v, None, n, base, rope_mode=kv.RopeMode.NONE)


def _room(rows):
    return (rows + 256 + 63) // 64 * 64


def prepare(case, seed):
    s = SHAPES[case["shape"]]
    hq, hkv, d, hybrid = s["hq"], s["hkv"], s["d"], case["shape"] == "hybrid"
    act = torch.float16 if case["act"] == "f16" else torch.float32
    layers, kind = case.get("layers", 1), case["kind"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(act)
    weight = lambda: 1.0 + 0.1 * torch.randn(d, generator=g, device="cuda")
    st = {"case": case, "scale": d ** -0.5, "hq": hq, "rope": s["rope"], "layers": layers}
    kv.set_launch_overlap(1)

    if kind in ("step", "decode"):
        ctx = case["context"]
        caches = Caches(case, _room(ctx), layers)
        _fill(case, caches.views, ctx - 1, g)
        st.update(caches=caches, k=rand(layers, hkv * d), v=rand(layers, hkv * d), w=weight() if hybrid else None,
                  out=torch.zeros(layers, hq, d, device="cuda"), ws=kv.decode_workspace(hq, d))
        if kind == "step":
            st.update(q=rand(layers, hq, d), gate=torch.randn(layers, hq, d, generator=g, device="cuda") if hybrid else None, position=ctx - 1)
            return st
        if hybrid:
            st.update(qfull=rand(layers, hq, 2 * d), q=torch.zeros(layers, hq, d, dtype=act, device="cuda"),
                      gate=torch.zeros(layers, hq, d, device="cuda"), qw=weight())
        else:
            st.update(q=rand(layers, hq, d))
        st["state"] = kv.make_decode_state(ctx - 1)
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            _decode_layers(st)
            stream.synchronize()
            st["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(st["graph"], stream=stream):
                _decode_layers(st)
        torch.cuda.current_stream().wait_stream(stream)
    elif kind == "batched":
        lengths = _lengths(case)
        sessions = [Caches(case, _room(n), layers) for n in lengths]
        for c, n in zip(sessions, lengths):
            _fill(case, c.views, n, g)
        splits, bound = kv.plan_batched_decode(lengths, hkv)
        st.update(sessions=sessions, q=rand(layers, len(lengths), hq, d), out=torch.zeros(layers, len(lengths), hq, d, device="cuda"),
                  lengths=torch.tensor(lengths, dtype=torch.int32, device="cuda"), ws=kv.decode_workspace(hq, d, len(lengths)),
                  tables=[kv.view_table(len(lengths)) for _ in range(layers)], splits=splits, bound=bound)
        for l in range(layers):     # the first step's calls fill the device-side view tables
            _batched_layer(st, l, [c.views[l] for c in sessions])
    elif kind == "prefill":
        p, t = case["prefix"], case["tokens"]
        caches = Caches(case, _room(p + t), layers)
        _fill(case, caches.views, p, g)
        st.update(caches=caches, k=rand(layers, t, hkv * d), v=rand(layers, t, hkv * d), q=rand(layers, t, hq, d), w=weight(),
                  gate=torch.randn(layers, t, hq, d, generator=g, device="cuda") if hybrid else None,
                  out=torch.zeros(layers, t, hq, d, device="cuda"), ws=kv.prefill_workspace(p + t, hkv, d, token_count=t, query_heads=hq))
    elif kind == "append":
        t = case["tokens"]
        st.update(caches=Caches(case, _room(t), layers), k=rand(layers, t, hkv * d), v=rand(layers, t, hkv * d), w=weight())
    else:
        n = case["prefix"]
        mode = kv.KvCacheQuantMode.kFp16Fp16 if case["cache"] == "f16" else kv.KvCacheQuantMode.kQ8Q8
        new = lambda: [kv.AttentionLayerKvCacheStorage(_room(n), mode, kv_heads=hkv, head_dim=d, qblock=32 if case["cache"] == "q8_0" else d)
                       for _ in range(layers)]
        src, dst = new(), new()
        _fill(case, [c.view() for c in src], n, g)
        rng = random.Random(seed)
        tokens = [rng.randrange(150000) for _ in range(n)]
        st.update(src=src, dst=dst, pool=kv.SnapshotPool(max_entries=8, max_bytes=3 << 30, granularity=1), tokens=tokens, prompt=tokens + [1, 2, 3])
    return st


def _decode_layers(st):
    hybrid = "qfull" in st
    for l, view in enumerate(st["caches"].views):
        if hybrid:
            kv.launch_q_split_norm_rope(st["qfull"][l], st["qw"], st["q"][l], st["gate"][l], 1, 0, heads=st["hq"], head_dim=view.head_dim,
                                        rope_mode=st["rope"], theta=THETA, decode_state=st["state"])
            kv.launch_decode_step(view, st["k"][l], st["v"][l], st["q"][l], query_heads=st["hq"], scale=st["scale"], decode_state=st["state"],
                                  k_norm_weight=st["w"], rope_mode=st["rope"], theta=THETA, gate=st["gate"][l], gated_output=st["out"][l],
                                  workspace=st["ws"])
        else:
            kv.launch_decode_step(view, st["k"][l], st["v"][l], st["q"][l], query_heads=st["hq"], scale=st["scale"], decode_state=st["state"],
                                  rope_mode=st["rope"], theta=THETA, output=st["out"][l], workspace=st["ws"])


def _batched_layer(st, l, views):
    kv.launch_decode_attention_batched(views, st["tables"][l], st["lengths"], st["bound"], st["q"][l], query_heads=st["hq"], scale=st["scale"],
                                       output=st["out"][l], workspace=st["ws"], num_splits=st["splits"])


def run(st):
    kind = st["case"]["kind"]
    if kind == "step":
        gate = st["gate"][0] if st["gate"] is not None else None
        kv.launch_decode_step(st["caches"].views[0], st["k"][0], st["v"][0], st["q"][0], query_heads=st["hq"], scale=st["scale"],
                              position=st["position"], k_norm_weight=st["w"], rope_mode=st["rope"], theta=THETA, gate=gate,
                              **({"output": st["out"][0]} if gate is None else {"gated_output": st["out"][0]}), workspace=st["ws"])
        return [st["out"]] + st["caches"].planes()
    if kind == "decode":
        st["graph"].replay()
        return [st["out"]] + st["caches"].planes()
    if kind == "batched":
        for l in range(st["layers"]):
            _batched_layer(st, l, None)
        return st["out"]
    if kind == "prefill":
        p, t = st["case"]["prefix"], st["case"]["tokens"]
        for l, view in enumerate(st["caches"].views):
            kv.launch_kv_store_quant(view, st["k"][l], st["v"][l], st["w"], t, p, rope_mode=st["rope"], theta=THETA)
            kv.launch_suffix_attention_quant(view, st["q"][l], st["gate"][l] if st["gate"] is not None else None, st["out"][l], st["ws"], t, p,
                                             query_heads=st["hq"], scale=st["scale"])
        return [st["out"]] + st["caches"].planes()
    if kind == "append":
        for l, view in enumerate(st["caches"].views):
            kv.launch_kv_store_quant(view, st["k"][l], st["v"][l], st["w"], st["case"]["tokens"], 0, rope_mode=st["rope"], theta=THETA)
        return st["caches"].planes()
    st["pool"].capture(st["tokens"], st["src"])
    st["pool"].restore(st["prompt"], st["dst"])
    return [t for c in st["dst"] for t in c.planes()]
