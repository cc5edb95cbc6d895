"""The work this library is measured on: single-GPU (one-rank) forms of its public entry points over the sizes they are
used at. `listed()` names the fixed cases, `draw()` gives more of the same ranges, `prepare()` builds what a program
holds before the call, `run()` is one call, `work()` what it cannot do without, `tolerance()` how far another correct
implementation of the same precision may be off, `exact()` the results in float64.

Kinds of case:
  decode   one decode step of paged GQA attention (plain op, its partial O||LSE form, or the sequence-parallel layer)
  linear   one tensor-parallel linear layer's GEMM (plain, column-parallel or row-parallel entry point)
  mlp      column-parallel linear, activation, row-parallel linear
  fp8      quantise the activations, then the block-scaled fp8 linear against weights quantised once
  a2a      MoE gate, low-latency fp8 dispatch, dequantisation for the experts, weighted combine (identity experts)
  ep_moe   the whole expert-parallel MoE block: gate, dispatch, two grouped GEMMs, combine
  moe_tp   tensor-parallel MoE: all-gather + grouped GEMM, activation, grouped GEMM + top-k reduce + reduce-scatter
"""
import math

import torch
import torch.nn.functional as F

from triton_distributed_b200.models import EPMoE, SpGQAFlashDecodeAttention, TPMLP
from triton_distributed_b200.ops import all_to_all, flash_decode, gemm, gemm_fp8, moe_tp, moe_utils
from triton_distributed_b200.runtime import LocalWorld

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
HEADS = ((16, 16), (32, 8), (64, 8), (6, 1), (96, 12))
MOST_FLOPS = 2.0 * 8192 * 49152 * 12288   # the largest listed case
MOST_BYTES = 4.5e9


def _decode(B, hq, hkv, head_dim, kv, page, dtype="bf16", ragged=False, soft_cap=0.0, entry="op"):
    return dict(kind="decode", B=B, hq=hq, hkv=hkv, head_dim=head_dim, kv=kv, page=page, dtype=dtype, ragged=ragged,
                soft_cap=soft_cap, entry=entry)


def listed():
    return [
        # one interactive request with a short context: launch latency and the merge of the splits decide
        dict(name="decode_b1_4k", **_decode(1, 32, 8, 128, 4096, 16)),
        # a serving batch whose sequences all have different lengths
        dict(name="decode_b32_ragged_8k", **_decode(32, 64, 8, 128, 8192, 64, dtype="fp16", ragged=True)),
        # a batch of long contexts through the sequence-parallel layer
        dict(name="decode_b8_32k", **_decode(8, 32, 8, 128, 32768, 16, entry="layer")),
        # one very long context: the KV cache is streamed once from HBM
        dict(name="decode_b1_1m", **_decode(1, 32, 8, 128, 1048576, 16)),
        # a decode step of 16 sequences through one rank's shard (1/8) of a large column-parallel layer
        dict(name="linear_m16", kind="linear", M=16, N=6144, K=12288, dtype="bf16", entry="gemm"),
        # a ragged prefill of a thousand tokens through half of an 11008-wide layer
        dict(name="linear_m1000", kind="linear", M=1000, N=5504, K=4096, dtype="fp16", entry="gemm_rs"),
        # the benchmark's headline layer on one GPU
        dict(name="ag_gemm_m8192", kind="linear", M=8192, N=49152, K=12288, dtype="bf16", entry="ag_gemm"),
        # a feed-forward block over a prefill of 2048 tokens
        dict(name="mlp_m2048", kind="mlp", M=2048, hidden=4096, ffn=14336, dtype="bf16", activation="gelu"),
        # a block-scaled fp8 layer over a large prefill, activations quantised on the fly
        dict(name="fp8_m8192", kind="fp8", M=8192, N=6144, K=4096, entry="ag_gemm"),
        # the low-latency all-to-all at its serving size
        dict(name="a2a_t128", kind="a2a", T=128, hidden=7168, E=256, topk=8),
        # the same tokens through one rank's 32 experts
        dict(name="ep_moe_t128", kind="ep_moe", T=128, hidden=7168, ffn=2048, E=32, topk=8),
        # a large prefill through a tensor-parallel MoE layer (1/8 of the intermediate size)
        dict(name="moe_tp_m8192", kind="moe_tp", M=8192, hidden=4096, inter=1792, E=8, topk=2),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread evenly over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, step * max(1, round(v / step)))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "linear", "linear", "mlp", "fp8", "a2a", "ep_moe", "moe_tp"))
    while True:
        if kind == "decode":
            hq, hkv = rng.choice(HEADS)
            case = _decode(_log(rng, 1, 64), hq, hkv, rng.choice((64, 128, 128, 256)), _log(rng, 1, 1 << 20),
                           rng.choice((1, 16, 16, 64)), rng.choice(("bf16", "fp16")), rng.random() < 0.5,
                           rng.choice((0.0, 0.0, 30.0)), rng.choice(("op", "layer", "partial")))
        elif kind == "linear":
            case = dict(kind=kind, M=_log(rng, 1, 8192), N=_log(rng, 256, 49152, 8), K=_log(rng, 128, 16384, 8),
                        dtype=rng.choice(("bf16", "fp16")), entry=rng.choice(("gemm", "ag_gemm", "gemm_rs")))
        elif kind == "mlp":
            case = dict(kind=kind, M=_log(rng, 1, 8192), hidden=_log(rng, 1024, 8192, 8), ffn=_log(rng, 1024, 28672, 8),
                        dtype=rng.choice(("bf16", "fp16")), activation=rng.choice(("gelu", "silu", "relu")))
        elif kind == "fp8":
            case = dict(kind=kind, M=_log(rng, 1, 8192), N=_log(rng, 256, 16384, 8), K=_log(rng, 128, 16384, 128),
                        entry=rng.choice(("gemm", "ag_gemm")))
        elif kind == "a2a":
            E = rng.choice((8, 32, 64, 128, 256))
            case = dict(kind=kind, T=_log(rng, 1, 2048), hidden=_log(rng, 256, 8192, 128), E=E, topk=rng.randint(1, 8))
        elif kind == "ep_moe":
            E = rng.choice((8, 16, 32, 60, 64))
            case = dict(kind=kind, T=_log(rng, 1, 2048), hidden=_log(rng, 512, 7168, 64), ffn=_log(rng, 256, 4096, 64),
                        E=E, topk=rng.randint(1, 8))
        else:
            E = rng.choice((8, 16, 32, 64))
            case = dict(kind=kind, M=_log(rng, 64, 8192), hidden=_log(rng, 256, 7168, 8), inter=_log(rng, 128, 3584, 8),
                        E=E, topk=rng.randint(1, 6))
        w = work(case)
        if w["flops"] <= MOST_FLOPS and w["bytes"] <= MOST_BYTES:
            return case


def _normal(gen, shape, dtype=torch.bfloat16, scale=1.0):
    t = torch.empty(shape, dtype=dtype, device="cuda").normal_(generator=gen)
    return t if scale == 1.0 else t.mul_(scale)


def _lens(case, gen):
    """Keys of every sequence: all `kv`, or evenly spread over (0, kv] in random order."""
    B, kv = case["B"], case["kv"]
    if not case["ragged"]:
        return torch.full((B,), kv, dtype=torch.int32, device="cuda")
    spread = torch.tensor([max(1, kv * (i + 1) // B) for i in range(B)], dtype=torch.int32, device="cuda")
    return spread[torch.randperm(B, generator=gen, device="cuda")]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    s = {"case": dict(case)}
    # one rank's symmetric buffers, owned by this state
    heap = LocalWorld(1, torch.device("cuda", torch.cuda.current_device())).heap(0)
    if kind == "decode":
        B, D, hkv, page, dt = case["B"], case["head_dim"], case["hkv"], case["page"], DTYPES[case["dtype"]]
        per_seq = -(-case["kv"] // page)
        s["q"] = _normal(gen, (B, case["hq"], D), dt)
        s["k"] = _normal(gen, (B * per_seq, page, hkv, D), dt)
        s["v"] = _normal(gen, (B * per_seq, page, hkv, D), dt)
        # pages as a running server hands them out: in no order
        s["table"] = torch.randperm(B * per_seq, generator=gen, device="cuda").to(torch.int32).view(B, per_seq)
        s["lens"] = _lens(case, gen)
        s["scale"] = D ** -0.5
        if case["entry"] == "layer":
            s["layer"] = SpGQAFlashDecodeAttention(0, 0, 1, 1, case["hq"], hkv, D, D, page, s["scale"], case["soft_cap"],
                                                   max_allowed_batch=B, heap=heap)
            s["lens"] = s["lens"].view(1, B)
    elif kind == "linear":
        M, N, K, dt = case["M"], case["N"], case["K"], DTYPES[case["dtype"]]
        s["a"], s["b"] = _normal(gen, (M, K), dt), _normal(gen, (N, K), dt, K ** -0.5)
        if case["entry"] == "ag_gemm":
            s["ctx"] = gemm.create_ag_gemm_intra_node_context(s["a"], s["b"], 0, 1, max_M=M, heap=heap)
        elif case["entry"] == "gemm_rs":
            s["ctx"] = gemm.create_gemm_rs_context(M, N, 0, 1, output_dtype=dt, heap=heap)
    elif kind == "mlp":
        M, H, I, dt = case["M"], case["hidden"], case["ffn"], DTYPES[case["dtype"]]
        s["x"] = _normal(gen, (M, H), dt)
        s["block"] = TPMLP(_normal(gen, (I, H), dt, H ** -0.5), _normal(gen, (H, I), dt, I ** -0.5), 0, 1, M,
                           activation=case["activation"], heap=heap)
    elif kind == "fp8":
        M, N, K = case["M"], case["N"], case["K"]
        s["x"] = _normal(gen, (M, K))
        s["b"], s["sb"] = gemm_fp8.quantize_fp8_blockwise(_normal(gen, (N, K), torch.bfloat16, K ** -0.5))
        if case["entry"] == "ag_gemm":
            s["ctx"] = gemm_fp8.create_ag_gemm_fp8_context(M, K, 0, 1, heap=heap)
    elif kind == "a2a":
        s["x"], s["logits"] = _normal(gen, (case["T"], case["hidden"])), _normal(gen, (case["T"], case["E"]), torch.float32)
        s["ctx"] = all_to_all.create_moe_dispatch_context(case["T"], case["hidden"], case["topk"], case["E"], 0, 1, heap=heap)
    elif kind == "ep_moe":
        H, I, E = case["hidden"], case["ffn"], case["E"]
        s["x"] = _normal(gen, (case["T"], H))
        s["block"] = EPMoE(_normal(gen, (E, H), torch.bfloat16, H ** -0.5), _normal(gen, (E, I, H), torch.bfloat16, H ** -0.5),
                           _normal(gen, (E, H, I), torch.bfloat16, I ** -0.5), case["topk"], 0, 1, case["T"], heap=heap)
    else:
        M, H, I, E, topk = case["M"], case["hidden"], case["inter"], case["E"], case["topk"]
        s["x"] = _normal(gen, (M, H))
        s["b1"], s["b2"] = _normal(gen, (E, H, I), torch.bfloat16, H ** -0.5), _normal(gen, (E, I, H), torch.bfloat16, I ** -0.5)
        ids, w = moe_utils.topk_softmax(_normal(gen, (M, E), torch.float32), topk, renormalize=True)
        s["ids"], s["w"] = ids, w
        s["up"] = moe_tp.create_ag_group_gemm_intra_node_context(None, s["x"], s["b1"], ids, E, max_M=M, rank=0, num_ranks=1,
                                                                 heap=heap)
        s["down"] = moe_tp.create_moe_rs_context(None, 0, 1, 1, M, H, E, topk, torch.bfloat16, torch.bfloat16, s["x"].device,
                                                 full_topk_ids=ids, full_topk_weight=w, heap=heap)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "decode":
        if case["entry"] == "layer":
            return s["layer"](s["q"], s["k"], s["v"], s["lens"], s["table"])
        op = flash_decode.gqa_fwd_batch_decode if case["entry"] == "op" else flash_decode.gqa_fwd_batch_decode_intra_rank
        return op(s["q"], s["k"], s["v"], None, None, s["lens"], s["table"], s["scale"], case["soft_cap"])
    if kind == "linear":
        if case["entry"] == "gemm":
            return gemm.gemm_persistent(s["a"], s["b"])
        return (gemm.ag_gemm_intra_node if case["entry"] == "ag_gemm" else gemm.gemm_rs)(s["a"], s["b"], s["ctx"])
    if kind in ("mlp", "ep_moe"):
        return s["block"](s["x"])
    if kind == "fp8":
        a, sa = gemm_fp8.quantize_fp8_rowwise(s["x"])
        if case["entry"] == "ag_gemm":
            return gemm_fp8.ag_gemm_fp8(a, sa, s["b"], s["sb"], s["ctx"])
        return gemm_fp8.gemm_fp8_blockscaled(a, sa, s["b"], s["sb"])
    if kind == "a2a":
        ids, w = moe_utils.topk_softmax(s["logits"], case["topk"])
        rows, scales, splits = all_to_all.moe_dispatch(s["ctx"], s["x"], ids, w)
        all_to_all.dequant_fp8(rows, scales, out=all_to_all.moe_expert_out_buffer(s["ctx"]))
        return {"rows": rows, "scales": scales, "splits": splits, "out": all_to_all.moe_combine(s["ctx"], None, splits)}
    h = moe_tp.ag_group_gemm_intra_node(s["x"], s["b1"], s["up"])
    return moe_tp.moe_reduce_rs(0, 1, 1, F.silu(h), s["b2"], s["down"])


def work(case):
    kind = case["kind"]
    if kind == "decode":
        B, kv, D = case["B"], case["kv"], case["head_dim"]
        keys = sum(max(1, kv * (i + 1) // B) for i in range(B)) if case["ragged"] else B * kv
        out = B * case["hq"] * (4 * (D + 1) if case["entry"] == "partial" else 2 * D)
        return {"bytes": 4.0 * keys * case["hkv"] * D + 2.0 * B * case["hq"] * D + out, "flops": 4.0 * keys * case["hq"] * D}
    if kind == "linear":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 2.0 * (M * K + N * K + M * N), "flops": 2.0 * M * N * K}
    if kind == "mlp":
        M, H, I = case["M"], case["hidden"], case["ffn"]
        return {"bytes": 2.0 * (2 * M * H + 2 * H * I), "flops": 4.0 * M * H * I}
    if kind == "fp8":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 2.0 * M * K + N * K + 4.0 * (-(-N // 128) * (K // 128)) + 2.0 * M * N, "flops": 2.0 * M * N * K}
    if kind == "a2a":
        T, H, topk = case["T"], case["hidden"], case["topk"]
        # tokens and logits in, fp8 rows with their scales out, the experts' bf16 rows once each way, the sums out
        rows = T * topk
        return {"bytes": 2.0 * T * H + 4.0 * T * case["E"] + 2.0 * rows * (H + H // 32) + 4.0 * rows * H + 2.0 * T * H, "flops": 4.0 * rows * H}
    if kind == "ep_moe":
        T, H, I, E, topk = case["T"], case["hidden"], case["ffn"], case["E"], case["topk"]
        used = min(E, T * topk)
        return {"bytes": 2.0 * (2 * T * H + E * H + 2 * used * H * I), "flops": 2.0 * T * E * H + 4.0 * T * topk * H * I}
    M, H, I, E, topk = case["M"], case["hidden"], case["inter"], case["E"], case["topk"]
    return {"bytes": 2.0 * (2 * M * H + 2 * E * H * I + 4 * M * topk * I), "flops": 4.0 * M * topk * H * I}


def tolerance(case):
    """About four times the distance measured between the path and a float64 statement of the same operation on the same
    inputs: the rounding of the 16-bit results (and of a 16-bit intermediate: attention probabilities, the activations
    between two GEMMs) is nearly all of it."""
    kind, fine = case["kind"], case.get("dtype") == "fp16"
    if kind == "decode" and case["entry"] == "partial":
        # fp32 results: the rounding of the probabilities, over a norm that the log-sum-exp column dominates
        return {"rel": 5e-4, "max": 4e-3} if fine else {"rel": 4e-3, "max": 2e-2}
    if kind == "decode":
        return {"rel": 1.1e-3, "max": 7.5e-3} if fine else {"rel": 9e-3, "max": 3e-2}
    if kind in ("linear", "fp8"):
        return {"rel": 8.5e-4, "max": 2e-3} if fine else {"rel": 7e-3, "max": 1.6e-2}
    if kind == "mlp":
        return {"rel": 1.6e-3, "max": 8e-3} if fine else {"rel": 1.25e-2, "max": 6e-2}
    if kind == "a2a":
        return {"rel": 9e-3, "max": 3e-2}
    return {"rel": 1.4e-2, "max": 8.5e-2}


def exact(case, seed):
    """What `run` returns for `prepare(case, seed)`, in float64 torch. fp8 operands are the quantised values themselves;
    16-bit intermediates (attention probabilities, activations between two GEMMs) are not rounded. None: an output that
    is the quantisation itself."""
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "decode":
        return _exact_decode(case, s)
    if kind == "linear":
        return s["a"].double() @ s["b"].double().t()
    if kind == "mlp":
        act = {"gelu": lambda h: F.gelu(h, approximate="tanh"), "silu": F.silu, "relu": F.relu}[case["activation"]]
        return act(s["x"].double() @ s["block"].w1.double().t()) @ s["block"].w2.double().t()
    if kind == "fp8":
        a, sa = _quantised(s["x"])
        sb = s["sb"].double().repeat_interleave(128, 0)[:case["N"]].repeat_interleave(128, 1)
        return (a.double() * sa.double().repeat_interleave(128, 1)) @ (s["b"].double() * sb).t()
    if kind == "a2a":
        p = torch.softmax(s["logits"].double(), -1)
        w = p.topk(case["topk"], -1).values
        q, scale = _quantised(s["x"])
        x = q.double() * scale.double().repeat_interleave(128, 1)
        return {"rows": None, "scales": None, "splits": None, "out": w.sum(-1, keepdim=True) * x}
    x, M = s["x"].double(), s["x"].shape[0]
    if kind == "ep_moe":
        block, E = s["block"], case["E"]
        p, ids = torch.softmax(x @ block.gate.double().t(), -1).topk(case["topk"], -1)
        w = p / p.sum(-1, keepdim=True)
        up = lambda e: block.w1[e].double().t()    # noqa: E731
        down = lambda e: block.w2[e].double().t()  # noqa: E731
    else:
        E, ids, w = case["E"], s["ids"].long(), s["w"].double()
        up, down = (lambda e: s["b1"][e].double()), (lambda e: s["b2"][e].double())
    out = torch.zeros((M, case["hidden"]), dtype=torch.float64, device="cuda")
    for e in range(E):
        tok, slot = torch.nonzero(ids == e, as_tuple=True)
        if tok.numel():
            out.index_add_(0, tok, (F.silu(x[tok] @ up(e)) @ down(e)) * w[tok, slot].unsqueeze(1))
    return out


def _quantised(x):
    """Per row and 128 values: the e4m3 values and their fp32 scale (largest magnitude / 448)."""
    g = x.float().view(x.shape[0], -1, 128)
    scale = g.abs().amax(-1).clamp_min(1e-12) / 448.0
    return (g / scale.unsqueeze(-1)).to(torch.float8_e4m3fn).view(x.shape), scale


def _exact_decode(case, s):
    B, hq, hkv, D, cap = case["B"], case["hq"], case["hkv"], case["head_dim"], case["soft_cap"]
    out = torch.empty((B, hq, D + 1), dtype=torch.float64, device="cuda")
    lens = s["lens"].view(B).tolist()
    for b in range(B):
        pages, n = s["table"][b].long(), lens[b]
        for h in range(hkv):
            heads = slice(h * hq // hkv, (h + 1) * hq // hkv)
            k = s["k"][pages, :, h].reshape(-1, D)[:n].double()
            v = s["v"][pages, :, h].reshape(-1, D)[:n].double()
            t = s["q"][b, heads].double() @ k.t() * s["scale"]
            if cap > 0:
                t = cap * torch.tanh(t / cap)
            out[b, heads, :D] = torch.softmax(t, -1) @ v
            out[b, heads, D] = torch.logsumexp(t, -1)
    return out if case["entry"] == "partial" else out[..., :D]
