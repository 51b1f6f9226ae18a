"""The work a user of this framework has it do, as timed cases: decode steps, batched products, prompts, mixture-of-experts
layers, row decodes and the smallest single calls, through the entry points of ``orome_b200.format``.

A case is a dict of plain values.  Its ``kind`` says which of the four paths it takes:

* ``dense``: transformer layers without attention -- q/k/v, output projection, gate/up + SwiGLU, down -- and, with
  ``vocab``, the lm_head and the arg-max of its logits.  ``batch`` 1 is a decode step: with ``norm`` the residual adds
  and the RMS norms either side of the products ride on them (``fuse_next``), with ``graph`` the step was captured once
  and is replayed, as a token loop does.  Larger batches are small batched decodes and prompts.
* ``product``: one matvec call.
* ``moe``: routing and the expert block (with ``shared`` also the shared expert) of mixture-of-experts layers.
* ``rows``: the decode of rows of a packed tensor to fp32 (the embedding lookup, and whole tensors).

Shapes of the listed cases are the benchmark's (9B and 27B sets, 35B-A3B-shape experts) or generic ones in between.
Weights are random blocks with the scales of trained tensors (standard deviation 0.03), activations are normal.
"""
import torch

from orome_b200 import format as F
from orome_b200 import synth

FORMATS = {"q8_0": synth.Q8_0, "q4_k": synth.Q4_K, "q5_k": synth.Q5_K, "q6_k": synth.Q6_K}
# format of attention and gate/up, of down, of the lm_head: single-format files, and the usual mixed ones
MIXES = {"q8_0": ("q8_0", "q8_0", "q8_0"), "q4_k": ("q4_k", "q4_k", "q4_k"), "q5_k": ("q5_k", "q5_k", "q5_k"), "q6_k": ("q6_k", "q6_k", "q6_k"),
         "q4_k_m": ("q4_k", "q6_k", "q6_k"), "q5_k_m": ("q5_k", "q6_k", "q6_k")}
# standard deviation of (weight / d) for uniform quants and scale fields, see _fill
UNIT_STD = {synth.Q8_0: 73.3, synth.Q4_K: 255.0, synth.Q5_K: 521.0, synth.Q6_K: 342.0}
WEIGHT_STD = 0.03
EPS = 1e-6


def listed():
    return [
        # one small projection issued on its own, where the call and the launch are the cost (k/v of a 2048-wide model)
        {"name": "call_q4_k_1024x2048", "kind": "product", "fmt": "q4_k", "rows": 1024, "cols": 2048, "batch": 1, "llama": False},
        # a decode token of the 9B-shape Q8_0 set, replayed as a graph, x at the width the benchmark uses
        {"name": "token_9b_q8_0", "kind": "dense", "mix": "q8_0", "hidden": 4096, "kv": 1024, "ffn": 12288, "layers": 32, "vocab": 151936,
         "batch": 1, "norm": True, "graph": True, "x_bits": 16, "llama": False},
        # a decode token of the 27B-shape mixed set (Q4_K, down and lm_head Q6_K), replayed as a graph
        {"name": "token_27b_q4_k_m", "kind": "dense", "mix": "q4_k_m", "hidden": 5120, "kv": 1024, "ffn": 17408, "layers": 64, "vocab": 151936,
         "batch": 1, "norm": True, "graph": True, "x_bits": 24, "llama": True},
        # decode layers of a small Q5_K model issued call by call, normalisation done by the caller
        {"name": "layers_q5_k_direct", "kind": "dense", "mix": "q5_k", "hidden": 2560, "kv": 512, "ffn": 9728, "layers": 4, "vocab": 0,
         "batch": 1, "norm": False, "graph": False, "x_bits": 24, "llama": False},
        # eight sequences decoded together on the 9B-shape layer
        {"name": "batch8_9b_q8_0", "kind": "dense", "mix": "q8_0", "hidden": 4096, "kv": 1024, "ffn": 12288, "layers": 2, "vocab": 0,
         "batch": 8, "norm": False, "graph": True, "x_bits": 24, "llama": False},
        # 64 rows at once on the 9B-shape layer in Q4_K: a large decode batch or a short prompt
        {"name": "batch64_9b_q4_k", "kind": "dense", "mix": "q4_k", "hidden": 4096, "kv": 1024, "ffn": 12288, "layers": 2, "vocab": 0,
         "batch": 64, "norm": False, "graph": False, "x_bits": 24, "llama": False},
        # a prompt of ordinary, odd length through a layer of the 27B-shape mixed set
        {"name": "prompt333_27b_q4_k_m", "kind": "dense", "mix": "q4_k_m", "hidden": 5120, "kv": 1024, "ffn": 17408, "layers": 1, "vocab": 0,
         "batch": 333, "norm": False, "graph": False, "x_bits": 24, "llama": True},
        # a long prompt through a layer of the 9B-shape set: the largest contraction
        {"name": "prompt2048_9b_q8_0", "kind": "dense", "mix": "q8_0", "hidden": 4096, "kv": 1024, "ffn": 12288, "layers": 1, "vocab": 0,
         "batch": 2048, "norm": False, "graph": False, "x_bits": 24, "llama": False},
        # one token through four 35B-A3B-shape expert layers (128 experts, top-8), replayed as a graph
        {"name": "moe_token", "kind": "moe", "hidden": 2048, "inter": 768, "experts": 128, "k": 8, "tokens": 1, "layers": 4, "shared": 0,
         "gate_up": "q4_k", "down": "q5_k", "graph": True},
        # 32 sequences decoded together through one such layer with a shared expert
        {"name": "moe_batch32_shared", "kind": "moe", "hidden": 2048, "inter": 768, "experts": 128, "k": 8, "tokens": 32, "layers": 1, "shared": 512,
         "gate_up": "q4_k", "down": "q5_k", "graph": False},
        # a prompt of odd length through one such layer
        {"name": "moe_prompt300", "kind": "moe", "hidden": 2048, "inter": 768, "experts": 128, "k": 8, "tokens": 300, "layers": 1, "shared": 0,
         "gate_up": "q4_k", "down": "q5_k", "graph": False},
        # rows of a packed tensor as fp32 (part of a token embedding)
        {"name": "rows_q6_k_5120x4096", "kind": "rows", "fmt": "q6_k", "rows": 5120, "cols": 4096, "llama": False},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over its logarithm."""
    v = lo * (hi / lo) ** rng.random()
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["product", "dense", "dense", "dense", "moe", "moe", "rows"])
    if kind == "product":
        fmt = rng.choice(sorted(FORMATS))
        return {"kind": kind, "fmt": fmt, "rows": _log(rng, 64, 65536), "cols": _log(rng, 256, 16384, 64 if fmt == "q8_0" and rng.random() < 0.3 else 256),
                "batch": rng.choice([1, 1, _log(rng, 2, 64)]), "llama": rng.random() < 0.3}
    if kind == "dense":
        batch = rng.choice([1, _log(rng, 2, 64), _log(rng, 64, 1152)])
        hidden = _log(rng, 1024, 5120, 256)
        return {"kind": kind, "mix": rng.choice(sorted(MIXES)), "hidden": hidden, "kv": rng.choice([256, 512, 1024]), "ffn": _log(rng, 2 * hidden, hidden * 7 // 512 * 256, 256),
                "layers": rng.randint(2, 6) if batch == 1 else 1, "vocab": 0 if batch > 1 or rng.random() < 0.6 else _log(rng, 8192, 151936),
                "batch": batch, "norm": batch == 1 and rng.random() < 0.6, "graph": batch <= 16 and rng.random() < 0.7,
                "x_bits": rng.choice([16, 24, 24]), "llama": rng.random() < 0.3}
    if kind == "moe":
        tokens = rng.choice([1, _log(rng, 2, 32), _log(rng, 32, 512)])
        return {"kind": kind, "hidden": _log(rng, 1024, 3072, 256), "inter": _log(rng, 512, 1536, 256), "experts": rng.choice([32, 64, 128]), "k": rng.choice([2, 4, 6, 8, 8]),
                "tokens": tokens, "layers": rng.randint(2, 4) if tokens == 1 else 1, "shared": rng.choice([0, 0, 512, 768]),
                "gate_up": rng.choice(["q4_k", "q4_k", "q5_k"]), "down": rng.choice(["q5_k", "q4_k", "q6_k"]), "graph": tokens <= 8 and rng.random() < 0.7}
    return {"kind": kind, "fmt": rng.choice(sorted(FORMATS)), "rows": _log(rng, 1, 8192), "cols": _log(rng, 1024, 8192, 256), "llama": rng.random() < 0.3}


# ---- inputs ---------------------------------------------------------------------------------------------------------------
def _fill(view, fmt, rows, cols, gen):
    """A packed tensor in place: every quant and scale pattern, block scales that give the weights their standard deviation."""
    nblk, bb = rows * (cols // synth.BLOCK_ELEMS[fmt]), synth.BLOCK_BYTES[fmt]
    v = view[:nblk * bb].random_(0, 256, generator=gen).view(nblk, bb)
    d = (torch.rand(nblk, generator=gen, device=view.device) * 0.8 + 0.6) * (WEIGHT_STD / UNIT_STD[fmt])
    half = lambda t: t.to(torch.float16).view(torch.uint8).view(nblk, 2)      # noqa: E731
    if fmt == synth.Q8_0:
        v[:, 0:2] = half(d)
    elif fmt == synth.Q6_K:
        v[:, 192:208] = (v[:, 192:208].view(torch.int8) >> 2).view(torch.uint8)       # sub-scales in [-32, 31]
        v[:, 208:210] = half(d)
    else:
        v[:, 0:2] = half(d)
        v[:, 2:4] = half(d * (7.5 if fmt == synth.Q4_K else 15.5))                  # mins centre the weights


class _Arena:
    """Packed tensors one behind the other in one allocation, as a model file holds them."""

    def __init__(self, tensors, gen, variant):
        offs, total = [], 0
        for _, fmt, rows, cols in tensors:
            offs.append(total)
            total += (synth.tensor_bytes(fmt, rows, cols) + 255) // 256 * 256
        self.mem = torch.empty(total + 256, dtype=torch.uint8, device="cuda")
        self.refs = {}
        for (name, fmt, rows, cols), off in zip(tensors, offs):
            _fill(self.mem[off:off + synth.tensor_bytes(fmt, rows, cols)], fmt, rows, cols, gen)
            self.refs[name] = F.tensor_ref(self.mem.data_ptr(), off, fmt, rows, cols, variant)


def _captured(issue):
    """`issue(stream)` run once and captured, as a token loop keeps its step."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        issue(side.cuda_stream)
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        issue(torch.cuda.current_stream().cuda_stream)
    return g


def _stream():
    return torch.cuda.current_stream().cuda_stream


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    state = {"product": _prepare_product, "dense": _prepare_dense, "moe": _prepare_moe, "rows": _prepare_rows}[case["kind"]](case, gen)
    if case.get("graph"):
        state["graph"] = _captured(state["issue"])
    return state


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda")


def _variant(case):
    return F.VARIANT_LLAMA if case["llama"] else F.VARIANT_DEFAULT


def _prepare_product(case, gen):
    fmt, rows, cols, batch = FORMATS[case["fmt"]], case["rows"], case["cols"], case["batch"]
    arena = _Arena([("w", fmt, rows, cols)], gen, _variant(case))
    ctx, x, y = F.Context(0), _randn(gen, batch, cols), torch.empty(batch, rows, device="cuda")
    ref = arena.refs["w"]

    def issue(stream):
        ctx.matvec(ref, x.data_ptr(), y.data_ptr(), batch, cols, rows, stream)
    return {"ctx": ctx, "keep": (arena, x), "issue": issue, "out": y}


def _dense_tensors(case):
    H, KV, A = case["hidden"], case["kv"], case["ffn"]
    main, down, head = (FORMATS[f] for f in MIXES[case["mix"]])
    out = []
    for l in range(case["layers"]):
        out += [(("q", l), main, H, H), (("k", l), main, KV, H), (("v", l), main, KV, H), (("o", l), main, H, H),
                (("gate", l), main, A, H), (("up", l), main, A, H), (("down", l), down, H, A)]
    return out + ([("head", head, case["vocab"], H)] if case["vocab"] else [])


def _prepare_dense(case, gen):
    H, KV, A, V, B, L = (case[k] for k in ("hidden", "kv", "ffn", "vocab", "batch", "layers"))
    arena = _Arena(_dense_tensors(case), gen, _variant(case))
    R = arena.refs
    ctx = F.Context(0)
    ctx.set_option(F.OPT_X_BITS, case["x_bits"])
    new = lambda *s: torch.zeros(*s, device="cuda")      # noqa: E731
    x, q, o, act, kv = _randn(gen, L, B, H), new(B, H), new(B, H), new(B, A), new(L, 2, B, KV)
    hid, logits, token = new(L, B, H), new(max(V, 1)), torch.zeros(1, dtype=torch.int32, device="cuda")
    seq = [R[n] for n, *_ in _dense_tensors(case)]
    parts, norms = new(2 * L + 1, 512), (_randn(gen, 2 * L + 1, max(H, 8)) * 0.1 + 1.0).to(torch.bfloat16)
    res = new(2 * L + 1, B, H)      # the residual stream after every add

    # without the fused norms the caller normalises, so every layer reads a unit-variance input of its own
    def decode_plain(stream):
        for l in range(L):
            src = x[l]
            ctx.hint_next(R["o", l])
            ctx.matvec_group([R["q", l], R["k", l], R["v", l]], src.data_ptr(), [q.data_ptr(), kv[l, 0].data_ptr(), kv[l, 1].data_ptr()], stream)
            ctx.hint_next(R["gate", l])
            ctx.matvec(R["o", l], q.data_ptr(), o.data_ptr(), 1, 0, 0, stream)
            ctx.hint_next(R["down", l])
            ctx.gate_up_swiglu(R["gate", l], R["up", l], o.data_ptr(), act.data_ptr(), 1, 0, 0, stream)
            ctx.hint_next(R["q", l + 1] if l + 1 < L else R.get("head"))
            ctx.matvec(R["down", l], act.data_ptr(), hid[l].data_ptr(), 1, 0, 0, stream)
        head(hid[L - 1], None, stream)

    def head(src, pro, stream):
        if V:
            if pro is not None:
                ctx.fuse_next(pro, None)
            ctx.matvec(R["head"], src.data_ptr(), logits.data_ptr(), 1, 0, 0, stream)
            ctx.argmax(logits.data_ptr(), V, token.data_ptr(), stream)

    # residual stream: res[0] is the embedded token (its sum of squares known to the caller), every o and down product adds to it
    pro = [F.NormPrologue(norms[i].data_ptr(), parts[i].data_ptr(), EPS) for i in range(2 * L + 1)]
    epi = [F.ResidualEpilogue(res[i].data_ptr(), parts[i + 1].data_ptr()) for i in range(2 * L)]
    res[0].copy_(x[0])
    parts[0, 0] = x[0].square().sum()

    def decode_norm(stream):
        for l in range(L):
            ctx.fuse_next(pro[2 * l], None)
            ctx.hint_next(R["o", l])
            ctx.matvec_group([R["q", l], R["k", l], R["v", l]], res[2 * l].data_ptr(), [q.data_ptr(), kv[l, 0].data_ptr(), kv[l, 1].data_ptr()], stream)
            ctx.fuse_next(None, epi[2 * l])
            ctx.hint_next(R["gate", l])
            ctx.matvec(R["o", l], q.data_ptr(), res[2 * l + 1].data_ptr(), 1, 0, 0, stream)
            ctx.fuse_next(pro[2 * l + 1], None)
            ctx.hint_next(R["down", l])
            ctx.gate_up_swiglu(R["gate", l], R["up", l], res[2 * l + 1].data_ptr(), act.data_ptr(), 1, 0, 0, stream)
            ctx.fuse_next(None, epi[2 * l + 1])
            ctx.hint_next(R["q", l + 1] if l + 1 < L else R.get("head"))
            ctx.matvec(R["down", l], act.data_ptr(), res[2 * l + 2].data_ptr(), 1, 0, 0, stream)
        head(res[2 * L], pro[2 * L], stream)

    def batched(stream):
        for l in range(L):
            src = x[l]
            for n, dst, rows in (("q", q, H), ("k", kv[l, 0], KV), ("v", kv[l, 1], KV)):
                ctx.matvec(R[n, l], src.data_ptr(), dst.data_ptr(), B, H, rows, stream)
            ctx.matvec(R["o", l], q.data_ptr(), o.data_ptr(), B, H, H, stream)
            ctx.gate_up_swiglu(R["gate", l], R["up", l], o.data_ptr(), act.data_ptr(), B, H, A, stream)
            ctx.matvec(R["down", l], act.data_ptr(), hid[l].data_ptr(), B, A, H, stream)

    if B > 1:
        out = {"kv": kv, "hidden": hid}
    else:
        out = {"kv": kv, "hidden": res if case["norm"] else hid}
        if V:
            out.update(logits=logits, token=token)
    return {"ctx": ctx, "keep": (arena, x, q, o, act, parts, norms, pro, epi, seq), "issue": batched if B > 1 else (decode_norm if case["norm"] else decode_plain), "out": out}


def _prepare_moe(case, gen):
    H, M, E, K, T, L, S = (case[k] for k in ("hidden", "inter", "experts", "k", "tokens", "layers", "shared"))
    gu, dn = FORMATS[case["gate_up"]], FORMATS[case["down"]]
    tensors = []
    for l in range(L):
        tensors += [(("gate", l), gu, E * M, H), (("up", l), gu, E * M, H), (("down", l), dn, E * H, M)]
        if S:
            tensors += [(("sgate", l), synth.Q8_0, S, H), (("sup", l), synth.Q8_0, S, H), (("sdown", l), synth.Q8_0, H, S)]
    arena = _Arena(tensors, gen, F.VARIANT_DEFAULT)
    R = arena.refs
    router, sgw = _randn(gen, L, E, H) / H ** 0.5, _randn(gen, L, H) / H ** 0.5
    ctx = F.Context(0)
    x = torch.zeros(L + 1, T, H, device="cuda")
    x[0] = _randn(gen, T, H)
    idx, w = torch.zeros(L, T, 8, dtype=torch.int32, device="cuda"), torch.zeros(L, T, 8, device="cuda")
    logits, slog = torch.empty(T, E + 1, device="cuda"), torch.empty(T, device="cuda")
    scratch = torch.empty(F.moe_block_scratch_floats(T, K, H, M, S), device="cuda")
    layers = []
    for l in range(L):
        proj = lambda n, fmt, rows, cols: F.ExpertProjRef(R[n, l].offset, synth.tensor_bytes(fmt, rows, cols), fmt)      # noqa: E731
        layers.append((F.ExpertLayerRef(arena.mem.data_ptr(), proj("gate", gu, M, H), proj("up", gu, M, H), proj("down", dn, H, M)),
                       F.tensor_ref(router[l].data_ptr(), 0, synth.F32, E, H), F.tensor_ref(sgw[l].data_ptr(), 0, synth.F32, 1, H),
                       (R["sgate", l], R["sup", l], R["sdown", l]) if S else None))

    def issue(stream):
        for l, (experts, rt, sg, shared) in enumerate(layers):
            src, iv, wv = x[l].data_ptr(), idx[l].data_ptr(), w[l].data_ptr()
            if shared:
                ctx.moe_route_pair(rt, sg, src, T, H, K, iv, wv, slog.data_ptr(), logits.data_ptr(), stream)
            else:
                ctx.moe_route(rt, src, T, H, K, iv, wv, logits.data_ptr(), stream)
            ctx.moe_block(experts, F.VARIANT_DEFAULT, shared, src, T, H, iv, wv, slog.data_ptr() if shared else 0, K, H, M, src, H, scratch.data_ptr(),
                          x[l + 1].data_ptr(), H, stream)
    return {"ctx": ctx, "keep": (arena, router, sgw, logits, slog, scratch), "issue": issue, "out": {"hidden": x, "idx": idx, "w": w}}


def _prepare_rows(case, gen):
    fmt, rows, cols = FORMATS[case["fmt"]], case["rows"], case["cols"]
    arena = _Arena([("w", fmt, rows, cols)], gen, _variant(case))
    ctx, out, ref = F.Context(0), torch.empty(rows, cols, device="cuda"), arena.refs["w"]

    def issue(stream):
        ctx.dequant_rows(ref, 0, rows, out.data_ptr(), stream)
    return {"ctx": ctx, "keep": arena, "issue": issue, "out": out}


def run(state):
    if "graph" in state:
        state["graph"].replay()
    else:
        state["issue"](_stream())
    return state["out"]


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "product":
        r, c, b = case["rows"], case["cols"], case["batch"]
        return {"bytes": synth.tensor_bytes(FORMATS[case["fmt"]], r, c) + 4 * b * (r + c), "flops": 2 * r * c * b}
    if kind == "rows":
        return {"bytes": synth.tensor_bytes(FORMATS[case["fmt"]], case["rows"], case["cols"]) + 4 * case["rows"] * case["cols"], "flops": 0}
    if kind == "dense":
        B, H, L, V = case["batch"], case["hidden"], case["layers"], case["vocab"]
        ts = _dense_tensors(case)
        io = L * B * 4 * (2 * H + 2 * case["kv"]) + 4 * V      # layer input and output, keys and values, logits
        return {"bytes": sum(synth.tensor_bytes(f, r, c) for _, f, r, c in ts) + io, "flops": 2 * B * sum(r * c for _, _, r, c in ts)}
    H, M, E, K, T, L, S = (case[k] for k in ("hidden", "inter", "experts", "k", "tokens", "layers", "shared"))
    hit = E * (1 - (1 - K / E) ** T)                            # expected number of experts that some token selects
    expert = 2 * synth.tensor_bytes(FORMATS[case["gate_up"]], M, H) + synth.tensor_bytes(FORMATS[case["down"]], H, M)
    other = 4 * E * H + 3 * (synth.tensor_bytes(synth.Q8_0, S, H) if S else 0) + 4 * T * 2 * H
    return {"bytes": L * (hit * expert + other), "flops": L * T * 2 * (3 * H * (K * M + S) + E * H)}


def tolerance(case):
    """Measured against an evaluation in fp64: four times the largest error seen in its class."""
    kind, batch = case["kind"], case.get("batch", 0)
    if kind == "rows":
        return "exact"
    if kind == "moe":
        # 24-bit x throughout: 4e-7; a shared expert's batched products have fp16 operands: 2e-4.  Tied logits may swap experts.
        return {"rel": 8e-4 if case["shared"] and case["tokens"] >= 4 else 4e-6, "differ": 0.002}
    if batch >= 4 and case.get("cols", 256) % 256 == 0:
        return {"rel": 2e-3 if kind == "product" else 5e-3}     # fp16 operands: 4.5e-4 a product, 1.2e-3 behind four of them
    if kind == "product":
        return {"rel": 1e-6}                                    # 24-bit x: 1.7e-7
    # 16-bit x: 2.1e-4 behind 32 layers; 24-bit x: 3e-6 behind 64 layers, 7e-6 where a layer's values span many decades
    return {"rel": 8e-4 if case["x_bits"] == 16 else 2e-5}
