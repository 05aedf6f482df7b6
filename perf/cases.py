"""The work that users of this framework have it do, as measurable cases: one pass of each through the public operators.

A pass is a decode step (up to 64 rows: replayed as a CUDA graph, as a serving loop does) or a piece of a prompt (more
rows: launched call by call) through the linear layers of the 27B-class decoder (hidden 5120; q|k|v 7168 x 5120,
o 5120 x 5120, gate|up 34816 x 5120, down 5120 x 17408) in one of the weight formats, a single Q8_0 projection, or the
vocabulary head.

    stack   W8A8, one scale per token and output channel: LinearStack, `layers` decoder layers with their quantizers
    q8      one Q8_0 projection with the file's own block scales: quant_rows(.., 32) and gemm(gk = 32)
    head    final norm and logits on Q8_0 weights: head_quant and head_q8
    w4a8    one layer of a Q4_K_M file: norm_g, rows_g and swiglu_g in front of the Q4_K / Q6_K projections
    mxfp4   one layer in MXFP4: quantize_act in front of each projection
"""
import types

import torch

from prism_b200 import decode, gguf_weights, linear_stack, mxfp4, quant, synth, w4a8, w8a8

HIDDEN, QKV, FFN, VOCAB = 5120, 7168, 17408, 248320
DECODE_ROWS = 64
EPS = 1e-6
LAYER = (("qkv", QKV, HIDDEN), ("o", HIDDEN, HIDDEN), ("gate_up", 2 * FFN, HIDDEN), ("down", HIDDEN, FFN))
LAYER_WEIGHTS = sum(n * k for _, n, k in LAYER)
# the k-quant kinds of a Q4_K_M file: V rows and down in Q6_K, the rest in Q4_K
KINDS = {"qkv": (("q4k", 6144), ("q6k", 1024)), "o": (("q4k", HIDDEN),), "gate_up": (("q4k", 2 * FFN),), "down": (("q6k", HIDDEN),)}
# the projections of a layer, and the slices that a rank of two or four holds
PROJECTIONS = ((7168, 5120), (5120, 5120), (34816, 5120), (5120, 17408), (3584, 5120), (5120, 2560), (17408, 5120),
               (5120, 8704), (1792, 5120), (8704, 5120), (5120, 4352))


def listed():
    return [
        {"name": "stack-1", "kind": "stack", "rows": 1, "layers": 4},            # one user's decode step
        {"name": "stack-16", "kind": "stack", "rows": 16, "layers": 4},          # a decode step of a small batch
        {"name": "stack-333", "kind": "stack", "rows": 333, "layers": 4},        # a short prompt of odd length
        {"name": "stack-8192", "kind": "stack", "rows": 8192, "layers": 4},      # a full prefill chunk
        {"name": "q8-16", "kind": "q8", "rows": 16, "n": 5120, "k": 5120},       # one projection call, latency
        {"name": "q8-500", "kind": "q8", "rows": 500, "n": 7168, "k": 5120},     # a prompt against the file's own scales
        {"name": "head-48", "kind": "head", "rows": 48, "n": VOCAB},             # logits of a busy decode batch
        {"name": "w4a8-12", "kind": "w4a8", "rows": 12},                         # decode on a Q4_K_M file
        {"name": "w4a8-50", "kind": "w4a8", "rows": 50},                         # the same with many users
        {"name": "w4a8-2048", "kind": "w4a8", "rows": 2048},                     # prefill on a Q4_K_M file
        {"name": "mxfp4-16", "kind": "mxfp4", "rows": 16},                       # decode in MXFP4
        {"name": "mxfp4-4000", "kind": "mxfp4", "rows": 4000},                   # prefill in MXFP4, odd length
    ]


def draw(rng):
    def rows(lo, hi):
        return min(hi, int(lo * (hi / lo + 1e-9) ** rng.random() + 0.5))
    kind = rng.choice(("stack", "stack", "q8", "head", "w4a8", "w4a8", "mxfp4"))
    if kind == "stack":
        return {"kind": kind, "rows": rows(1, 8192), "layers": rng.randint(1, 4)}
    if kind == "q8":
        n, k = rng.choice(PROJECTIONS)
        return {"kind": kind, "rows": rows(1, 1024), "n": n, "k": k}
    if kind == "head":
        return {"kind": kind, "rows": rows(1, 64), "n": VOCAB // rng.choice((1, 2, 4))}
    return {"kind": kind, "rows": rows(1, 4096)}


def _activations(rows, cols, gen, dtype=torch.bfloat16):
    """N(0, 1) with eight outlier channels, as the inputs of a decoder's projections have."""
    x = torch.randn(rows, cols, generator=gen, device="cuda")
    x[:, torch.randint(0, cols, (8,), generator=gen, device="cuda")] *= 20.0
    return x.to(dtype)


def _q8_weight(n, k, gen):
    """N(0, 0.02^2) weights as Q8_0: int8 [n, k] and the blocks' scales fp32 [n, k / 32]."""
    q, s = torch.empty(n, k, dtype=torch.int8, device="cuda"), torch.empty(n, k // 32, device="cuda")
    for r in range(0, n, 16384):
        w = torch.randn(min(16384, n - r), k, generator=gen, device="cuda") * 0.02
        q[r:r + 16384], s[r:r + 16384] = w8a8.weight_from_q8(synth.q8_0(w), 32)
    return q, s


def _k_quants(kind, n, k, gen, pools):
    """A k-quant matrix of N(0, 0.02^2) weights: its super-blocks drawn from a pool that was quantized on the host."""
    pool = pools[kind]
    at = torch.randint(0, pool.shape[0], (n * (k // 256),), generator=gen, device="cuda")
    which = gguf_weights.GGML_Q4_K if kind == "q4k" else gguf_weights.GGML_Q6_K
    return gguf_weights.KQuant(pool[at].reshape(n, k // 256, pool.shape[1]), which, k)


def _graph(step):
    """`step` as a decode loop runs it: once eagerly, then captured; the replay."""
    step()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    return graph.replay


def prepare(case, seed):
    kind, rows = case["kind"], case["rows"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    st = types.SimpleNamespace(kind=kind, rows=rows, n_rows=torch.tensor([rows], dtype=torch.int32, device="cuda"))
    if kind == "stack":
        layers = [linear_stack.make_layer_weights(i, "cuda", seed_cfg=1 + seed % 1000003) for i in range(case["layers"])]
        st.stack = linear_stack.LinearStack(layers, rows, "cuda")
        st.h0 = torch.randn(rows, HIDDEN, generator=gen, device="cuda")
        st.step = lambda: st.stack(st.h0)
        st.out = st.stack.h
    elif kind == "q8":
        st.w, st.ws = _q8_weight(case["n"], case["k"], gen)
        st.x = _activations(rows, case["k"], gen)
        st.out = torch.empty(rows, case["n"], dtype=torch.bfloat16, device="cuda")
        st.step = lambda: _q8_step(st)
    elif kind == "head":
        st.w, s = _q8_weight(case["n"], HIDDEN, gen)
        st.ws = s.to(torch.float16).float()
        st.h = _activations(rows, HIDDEN, gen, torch.float32)
        st.norm = 1.0 + 0.1 * torch.randn(HIDDEN, generator=gen, device="cuda")
        st.q = torch.empty(rows, HIDDEN, dtype=torch.int8, device="cuda")
        st.s = torch.empty(rows, HIDDEN // 32, device="cuda")
        st.out = torch.empty(rows, case["n"], device="cuda")
        st.step = lambda: _head_step(st)
    else:
        (_prepare_w4a8 if kind == "w4a8" else _prepare_mxfp4)(st, seed, gen)
        step = _w4a8_step if kind == "w4a8" else _mxfp4_step
        st.step = lambda: step(st)
    if rows <= DECODE_ROWS and kind not in ("q8", "head"):
        st.step = _graph(st.step)
    return st


def _layer_buffers(st, gen):
    """The residual, the layer's bf16 inputs and outputs."""
    rows = st.rows
    st.h0 = _activations(rows, HIDDEN, gen, torch.float32)
    st.h = torch.empty_like(st.h0)
    st.attn = _activations(rows, HIDDEN, gen)
    st.qkv = torch.empty(rows, QKV, dtype=torch.bfloat16, device="cuda")
    st.gu = torch.empty(rows, 2 * FFN, dtype=torch.bfloat16, device="cuda")
    st.out = {"qkv": st.qkv, "gate_up": st.gu, "h": st.h}


def _prepare_w4a8(st, seed, gen):
    host = torch.Generator().manual_seed(seed)
    w = torch.randn(4096, 256, generator=host) * 0.02
    pools = {"q4k": synth.q4_k(w).raw.reshape(4096, -1).cuda(), "q6k": synth.q6_k(w).raw.reshape(4096, -1).cuda()}
    st.w = {name: w4a8.segments([_k_quants(kind, n, k, gen, pools) for kind, n in KINDS[name]], "cuda") for name, _, k in LAYER}
    _layer_buffers(st, gen)
    st.norm = 1.0 + 0.1 * torch.randn(2, HIDDEN, generator=gen, device="cuda")
    st.act = {k: (torch.empty(st.rows, k, dtype=torch.int8, device="cuda"), torch.empty(k // 256, st.rows, device="cuda"),
                  torch.empty(k // 256, st.rows, 16, dtype=torch.int8, device="cuda")) for k in (HIDDEN, FFN)}


def _prepare_mxfp4(st, seed, gen):
    host = torch.Generator().manual_seed(seed)
    pool = mxfp4.pack(torch.randn(65536, 32, generator=host) * 0.02)
    pq, ps = pool.q.cuda(), pool.s.cuda()
    st.w = {}
    for name, n, k in LAYER:
        at = torch.randint(0, pq.shape[0], (n * (k // 32),), generator=gen, device="cuda")
        st.w[name] = mxfp4.prepare(mxfp4.MX4(pq[at].reshape(n, k // 2), ps[at].reshape(n, k // 32), n, k))
    _layer_buffers(st, gen)
    st.ffn = _activations(st.rows, FFN, gen)
    st.act = {k: (torch.empty(st.rows, k // 2, dtype=torch.uint8, device="cuda"),
                  torch.empty(st.rows, k // 32, dtype=torch.uint8, device="cuda")) for k in (HIDDEN, FFN)}


def _q8_step(st):
    q, s = w8a8.quant_rows(st.x, 32, st.n_rows)
    w8a8.gemm(q, s, st.w, st.ws, st.out, st.n_rows, 32)


def _head_step(st):
    decode.head_quant(st.h, st.norm, st.q, st.s, st.n_rows, st.rows, EPS)
    decode.head_q8(st.q, st.s, st.w, st.ws, st.out, st.n_rows, st.rows)


def _w4a8_step(st):
    rows, n = st.rows, st.n_rows
    (q, s, xs), (fq, fs, fxs) = st.act[HIDDEN], st.act[FFN]
    st.h.copy_(st.h0)
    quant.norm_g(st.h, st.norm[0], q, s, xs, n, rows, EPS)
    w4a8.gemm_segs(q, s, xs, st.w["qkv"], st.qkv, n)
    quant.rows_g(st.attn, q, s, xs, n, rows)
    w4a8.gemm_segs(q, s, xs, st.w["o"], st.h, n, epi=1)
    quant.norm_g(st.h, st.norm[1], q, s, xs, n, rows, EPS)
    w4a8.gemm_segs(q, s, xs, st.w["gate_up"], st.gu, n)
    quant.swiglu_g(st.gu, fq, fs, fxs, n, rows)
    w4a8.gemm_segs(fq, fs, fxs, st.w["down"], st.h, n, epi=1)


def _mxfp4_step(st):
    rows = st.rows
    (q, s), (fq, fs) = st.act[HIDDEN], st.act[FFN]
    st.h.copy_(st.h0)
    mxfp4.quantize_act(st.h, q, s)
    mxfp4.gemm(q, s, st.w["qkv"], st.qkv, rows)
    mxfp4.quantize_act(st.attn, q, s)
    mxfp4.gemm(q, s, st.w["o"], st.h, rows, epi=1)
    mxfp4.quantize_act(st.h, q, s)
    mxfp4.gemm(q, s, st.w["gate_up"], st.gu, rows)
    mxfp4.quantize_act(st.ffn, fq, fs)
    mxfp4.gemm(fq, fs, st.w["down"], st.h, rows, epi=1)


def run(state):
    state.step()
    return state.out


def work(case):
    """Weights at the density of their file format, once; the pass's inputs and outputs, once."""
    kind, m = case["kind"], case["rows"]
    if kind == "stack":
        return {"bytes": case["layers"] * (LAYER_WEIGHTS + 4 * sum(n for _, n, _ in LAYER)) + 8 * m * HIDDEN,
                "flops": 2 * m * case["layers"] * LAYER_WEIGHTS}
    if kind == "q8":
        return {"bytes": case["n"] * case["k"] * 34 / 32 + 2 * m * (case["n"] + case["k"]), "flops": 2 * m * case["n"] * case["k"]}
    if kind == "head":
        return {"bytes": case["n"] * HIDDEN * 34 / 32 + 4 * m * (case["n"] + HIDDEN), "flops": 2 * m * case["n"] * HIDDEN}
    outer = m * (8 * HIDDEN + 2 * HIDDEN + 2 * QKV + 4 * FFN)
    if kind == "mxfp4":
        return {"bytes": LAYER_WEIGHTS * 17 / 32 + outer + 2 * m * FFN, "flops": 2 * m * LAYER_WEIGHTS}
    weights = sum(n * k * (144 if t == "q4k" else 210) / 256 for name, _, k in LAYER for t, n in KINDS[name])
    return {"bytes": weights + outer, "flops": 2 * m * LAYER_WEIGHTS}


def tolerance(case):
    """Measured against the same pass with norms and SwiGLU in 64 bits (and, for mxfp4, the products too), times four.
    What differs there is the odd int8 value on a rounding boundary and the bf16 rounding of what follows from it."""
    return {"stack": {"rel": 3e-2},        # 0 up to 16 rows, 9.7e-3 at 700: four layers without a norm square what a row holds
            "q8": "exact",                 # integer sums, then single fp32 operations in a stated order
            "head": {"rel": 1e-4},         # 1.4e-7 with every int8 value alike; one value's step is 2e-5
            "w4a8": {"rel": 1.2e-3},       # 3.1e-4 at 500 rows
            "mxfp4": {"rel": 1e-3},        # 0: a one-ulp bf16 difference of an output in a thousand would be 1e-4
            }[case["kind"]]
