"""What is timed when this library is measured: the calls that a DiT with 2048 channels (16 heads of 128) makes on its
attention path, through the public entry points of kiln_b200.ops, over the sizes that image generation and LoRA training
reach (256 to 4096 image tokens, contexts of 16 to 512 text tokens).

Kinds of case:
  self      one block's self-attention; with norm=True the per-head Q/K RMSNorm and the rotary embedding run in the call
  cross     one block's attention to a text context, padded analytically to 512 keys
  nag       the same against a positive and a negative context with the guidance combine
  cross_kv  the once-per-prompt producer of one block's cross-attention K and V
  block     the attention half of a block on fp16 activations: q, k, v projections with the head epilogue, self-attention,
            output projection into the residual stream, cross-attention query projection, nag attention, output projection;
            lora > 0 adds an unmerged LoRA of that stacked rank to the q, k, v projections
  mlp       the other two linear layers of a block: up-projection with GELU, gated down-projection into the residual stream
  bwd       attention gradients of a training step: of self-attention, and with ctx > 0 of the block's cross-attention too
"""
import math

import torch

from kiln_b200 import ops

H, D = 16, 2048            # heads, channels
CTX_CHANNELS = 1024        # width of the text encoder's output
CTX_LEN = 512              # padded context length
MLP = 4 * D
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
NAG = (5.0, 2.5, 0.25)     # scale, tau, alpha


def listed():
    return [
        # a short prompt's cross-attention at 512x768: the smallest call of a step, a latency chain
        {"name": "cross_1536_ctx26_f16", "kind": "cross", "tokens": 1536, "batch": 1, "dtype": "f16", "ctx": 26},
        # K and V of a full-length context for one block, from the text encoder's fp32 output
        {"name": "cross_kv_512_f32", "kind": "cross_kv", "tokens": 512, "batch": 1, "dtype": "f32"},
        # a token count that no tile divides, on fp32 activations that were normalised and rotated before the call
        {"name": "self_1000_f32", "kind": "self", "tokens": 1000, "batch": 1, "dtype": "f32", "norm": False},
        # self-attention of a 512x768 image
        {"name": "self_1536_bf16", "kind": "self", "tokens": 1536, "batch": 1, "dtype": "bf16", "norm": True},
        # self-attention of a 1024x1024 image
        {"name": "self_4096_bf16", "kind": "self", "tokens": 4096, "batch": 1, "dtype": "bf16", "norm": True},
        # both halves of classifier-free guidance at 768x1152
        {"name": "self_cfg_2x3456_bf16", "kind": "self", "tokens": 3456, "batch": 2, "dtype": "bf16", "norm": True},
        # guidance against a long positive and a short negative prompt at 512x768, K and V cached in fp16
        {"name": "nag_1536_ctx378_168_f16", "kind": "nag", "tokens": 1536, "batch": 1, "dtype": "f16", "ctx": 378, "ctx_neg": 168},
        # guidance with both contexts full at 1024x1024
        {"name": "nag_4096_ctx512_512_bf16", "kind": "nag", "tokens": 4096, "batch": 1, "dtype": "bf16", "ctx": 512, "ctx_neg": 512},
        # the attention half of a block at 512x768 with an unmerged LoRA on q, k, v
        {"name": "block_1536_lora32_f16", "kind": "block", "tokens": 1536, "batch": 1, "dtype": "f16", "ctx": 77, "ctx_neg": 26, "lora": 32},
        # the MLP of a block at 768x1152
        {"name": "mlp_3456_f16", "kind": "mlp", "tokens": 3456, "batch": 1, "dtype": "f16"},
        # a training step's attention gradients of one block at 512x512, fp32 activations as the trainer has them
        {"name": "bwd_1024_ctx77_f32", "kind": "bwd", "tokens": 1024, "batch": 1, "dtype": "f32", "ctx": 77},
        # self-attention gradients at 1024x1024: the largest call
        {"name": "bwd_4096_bf16", "kind": "bwd", "tokens": 4096, "batch": 1, "dtype": "bf16", "ctx": 0},
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["cross", "cross_kv", "self", "self", "self", "nag", "nag", "block", "mlp", "bwd", "bwd"])
    c = {"kind": kind, "tokens": spread(256, 4096), "batch": 1, "dtype": rng.choice(["f16", "bf16", "f32"])}
    if kind == "self":
        c["norm"] = rng.random() < 0.7
        if c["tokens"] <= 3456 and rng.random() < 0.3:
            c["batch"] = 2
    elif kind == "cross":
        c["ctx"] = spread(16, CTX_LEN)
    elif kind == "nag":
        c["ctx"], c["ctx_neg"] = spread(16, CTX_LEN), spread(16, CTX_LEN)
    elif kind == "cross_kv":
        c["tokens"] = spread(16, CTX_LEN)
    elif kind == "block":
        c["dtype"] = "f16"
        c["tokens"] = spread(256, 4096)
        c["ctx"], c["ctx_neg"] = spread(16, CTX_LEN), spread(16, CTX_LEN)
        c["lora"] = rng.choice([0, 0, 16, 32, 72])
    elif kind == "mlp":
        c["dtype"] = "f16"
    elif kind == "bwd":
        c["ctx"] = rng.choice([0, spread(16, CTX_LEN)])
    return c


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    T, B, kind = case["tokens"], case["batch"], case["kind"]

    def normal(rows, cols, dtype=dt, std=1.0):
        return (torch.randn(rows, cols, generator=gen, device="cuda") * std).to(dtype)

    def empty(rows, cols, dtype):
        return torch.empty(rows, cols, dtype=dtype, device="cuda")

    def norm_weight():
        return (1.0 + 0.02 * torch.randn(128, generator=gen, device="cuda")).to(torch.bfloat16)

    def scratch(n):
        return torch.empty(max(int(n), 16), dtype=torch.uint8, device="cuda")

    def linear_weight(n, k):
        return normal(n, k, torch.float16, 1.0 / math.sqrt(k))

    def rope(n):
        # two image axes of 32 frequencies each on a grid as square as n allows
        w = max(1, int(math.sqrt(n)))
        pos = torch.arange(n, device="cuda")
        freq = 10000.0 ** (-torch.arange(32, device="cuda") / 32.0)
        ang = torch.cat([(pos // w)[:, None] * freq, (pos % w)[:, None] * freq], dim=1)
        return ang.cos().contiguous(), ang.sin().contiguous()

    s = {"case": case}
    out_dt = torch.float16 if dt == torch.float32 else dt
    if kind == "self":
        s["q"], s["k"], s["v"] = (normal(B * T, D) for _ in range(3))
        s["out"] = empty(B * T, D, out_dt)
        if case["norm"]:
            s["qn"], s["kn"] = norm_weight(), norm_weight()
            s["cos"], s["sin"] = rope(T)
        s["ws"] = scratch(ops.workspace_bytes(B * T, B * T, H, dt, case["norm"], case["norm"]))
    elif kind == "cross":
        s["q"], s["qn"] = normal(T, D), norm_weight()
        s["k"], s["v"] = normal(case["ctx"], D), normal(case["ctx"], D)
        s["out"] = empty(T, D, out_dt)
        s["ws"] = scratch(ops.workspace_bytes(T, case["ctx"], H, dt, True, False))
    elif kind == "nag":
        s["q"], s["qn"] = normal(T, D), norm_weight()
        s["kp"], s["vp"] = normal(case["ctx"], D), normal(case["ctx"], D)
        s["kn"], s["vn"] = normal(case["ctx_neg"], D), normal(case["ctx_neg"], D)
        s["out"] = empty(T, D, out_dt)
        s["ws"] = scratch(ops.workspace_bytes(T, max(case["ctx"], case["ctx_neg"]), H, dt, True, False, n_ctx=2))
    elif kind == "cross_kv":
        s["ctx"] = normal(T, CTX_CHANNELS)
        s["wk"], s["wv"], s["kn"] = linear_weight(D, CTX_CHANNELS), linear_weight(D, CTX_CHANNELS), norm_weight()
        s["k"], s["v"] = empty(T, D, torch.float16), empty(T, D, torch.float16)
        s["ws"] = scratch(T * CTX_CHANNELS * 2)
    elif kind == "block":
        s["x1"], s["x2"] = normal(T, D), normal(T, D)          # the normalised, modulated inputs of the two attentions
        s["res"] = normal(T, D, torch.float32)                 # the residual stream
        s["w"] = [linear_weight(D, D) for _ in range(6)]       # q, k, v, o of self-attention; q, o of cross-attention
        s["qn"], s["kn"], s["cqn"] = norm_weight(), norm_weight(), norm_weight()
        s["cos"], s["sin"] = rope(T)
        s["gate"] = (0.1 * torch.randn(2, D, generator=gen, device="cuda"))
        s["kp"], s["vp"] = normal(case["ctx"], D), normal(case["ctx"], D)
        s["kneg"], s["vneg"] = normal(case["ctx_neg"], D), normal(case["ctx_neg"], D)
        s["qkv"] = [empty(T, D, torch.float16) for _ in range(3)]
        s["a"], s["cq"], s["ca"] = (empty(T, D, torch.float16) for _ in range(3))
        if case["lora"]:
            r = case["lora"]
            s["la"] = linear_weight(3 * r, D)                  # the three down-projections stacked
            s["lb"] = [normal(D, r, torch.float16, 0.5 / math.sqrt(r)) for _ in range(3)]
            s["t"] = empty(T, 3 * r, torch.float16)
        s["ws"] = scratch(ops.workspace_bytes(T, T, H, torch.float16))
        s["ws2"] = scratch(ops.workspace_bytes(T, max(case["ctx"], case["ctx_neg"]), H, torch.float16, n_ctx=2))
    elif kind == "mlp":
        s["x"], s["res"] = normal(T, D), normal(T, D, torch.float32)
        s["w1"], s["w2"] = linear_weight(MLP, D), linear_weight(D, MLP)
        s["gate"] = (0.1 * torch.randn(D, generator=gen, device="cuda"))
        s["h"] = empty(T, MLP, torch.float16)
    elif kind == "bwd":
        s["calls"] = []
        for tk, npad in [(T, 0)] + ([(case["ctx"], CTX_LEN - case["ctx"])] if case["ctx"] else []):
            t = {"tk": tk, "npad": npad, "q": normal(B * T, D), "k": normal(B * tk, D), "v": normal(B * tk, D), "do": normal(B * T, D)}
            t["dq"], t["dk"], t["dv"] = empty(B * T, D, torch.float32), empty(B * tk, D, torch.float32), empty(B * tk, D, torch.float32)
            s["calls"].append(t)
        s["ws"] = scratch(max(ops.lib().kb_attn_bwd_workspace_bytes(B, T, t["tk"], H, {"f16": 0, "bf16": 1, "f32": 2}[case["dtype"]])
                              for t in s["calls"]))
    return s


def run(s):
    case = s["case"]
    T, B, kind = case["tokens"], case["batch"], case["kind"]
    if kind == "self":
        return ops.attn_self(s["out"], s["q"], s["k"], s["v"], B, T, H, qn_w=s.get("qn"), kn_w=s.get("kn"), rope_cos=s.get("cos"),
                             rope_sin=s.get("sin"), workspace=s["ws"])
    if kind == "cross":
        return ops.attn_cross(s["out"], s["q"], s["k"], s["v"], T, case["ctx"], CTX_LEN - case["ctx"], H, qn_w=s["qn"], workspace=s["ws"])
    if kind == "nag":
        return ops.attn_nag(s["out"], s["q"], s["kp"], s["vp"], case["ctx"], CTX_LEN - case["ctx"], s["kn"], s["vn"], case["ctx_neg"],
                            CTX_LEN - case["ctx_neg"], *NAG, T, H, qn_w=s["qn"], workspace=s["ws"])
    if kind == "cross_kv":
        return ops.cross_kv(s["k"], s["v"], s["ctx"], s["wk"], s["wv"], kn_w=s["kn"], workspace=s["ws"])
    if kind == "block":
        w, r = s["w"], case["lora"]
        loras = None
        if r:
            ops.linear16(s["t"], s["x1"], s["la"], ops.EPI_F16)
            loras = [(s["t"][:, i * r:(i + 1) * r], s["lb"][i]) for i in range(3)]
        q, k, v = ops.linear16_qkv(s["qkv"], s["x1"], w[:3], (s["qn"], s["kn"], None), rope_cos=s["cos"], rope_sin=s["sin"], loras=loras)
        ops.attn_self(s["a"], q, k, v, B, T, H, workspace=s["ws"])
        ops.linear16(s["res"], s["a"], w[3], ops.EPI_RESID, gate=s["gate"][0])
        ops.linear16(s["cq"], s["x2"], w[4], ops.EPI_HEADS16, head_w=s["cqn"])
        ops.attn_nag(s["ca"], s["cq"], s["kp"], s["vp"], case["ctx"], CTX_LEN - case["ctx"], s["kneg"], s["vneg"], case["ctx_neg"],
                     CTX_LEN - case["ctx_neg"], *NAG, T, H, workspace=s["ws2"])
        ops.linear16(s["res"], s["ca"], w[5], ops.EPI_RESID, gate=s["gate"][1])
        return q, k, v, s["a"], s["ca"], s["res"]
    if kind == "mlp":
        ops.linear16(s["h"], s["x"], s["w1"], ops.EPI_GELU16)
        return s["h"], ops.linear16(s["res"], s["h"], s["w2"], ops.EPI_RESID, gate=s["gate"])
    if kind == "bwd":
        return [ops.attn_bwd(t["dq"], t["dk"], t["dv"], t["q"], t["k"], t["v"], t["do"], B, T, t["tk"], t["npad"], H, workspace=s["ws"])
                for t in s["calls"]]
    raise ValueError(kind)


def work(case):
    T, B, kind = case["tokens"], case["batch"], case["kind"]
    e = {"f16": 2, "bf16": 2, "f32": 4}[case["dtype"]]
    ctx, ctx_neg, lora = case.get("ctx", 0), case.get("ctx_neg", 0), case.get("lora", 0)
    attn = 4.0 * T * D                                          # flops of one attention per image and key
    if kind == "self":
        tables = 2 * T * 64 * 4 if case["norm"] else 0
        return {"bytes": B * T * D * (3 * e + 2) + tables, "flops": B * attn * T}
    if kind in ("cross", "nag"):
        return {"bytes": T * D * (e + 2) + 2 * (ctx + ctx_neg) * D * e, "flops": attn * (ctx + ctx_neg)}
    if kind == "cross_kv":
        return {"bytes": T * CTX_CHANNELS * e + 2 * D * CTX_CHANNELS * 2 + 2 * T * D * 2, "flops": 2 * 2.0 * T * D * CTX_CHANNELS}
    if kind == "block":
        # read: both inputs, the residual stream, weights, contexts, LoRA; written: q, k, v, both attentions, the residual stream
        return {"bytes": T * D * (2 * 2 + 4 + 5 * 2 + 4) + 6 * D * D * 2 + 2 * (ctx + ctx_neg) * D * 2 + 6 * D * lora * 2,
                "flops": 6 * 2.0 * T * D * D + attn * (T + ctx + ctx_neg) + 2 * 2.0 * T * D * 3 * lora}
    if kind == "mlp":
        return {"bytes": T * D * (2 + 4 + 4) + T * MLP * 2 + 2 * D * MLP * 2, "flops": 2 * 2.0 * T * D * MLP}
    keys = [T] + ([ctx] if ctx else [])
    return {"bytes": sum(B * (2 * T + 2 * k) * D * e + B * (T + 2 * k) * D * 4 for k in keys), "flops": sum(2.5 * B * attn * k for k in keys)}


def tolerance(case):
    # About four times the error measured against a float64 evaluation on the same inputs: fp16 operands with fp32 sums give
    # 2e-4 on plain products, 3e-4 behind the head norm, 3e-4 to 5e-4 on attention and its gradients (worst with fp32 inputs,
    # which are rounded to fp16 first); a bf16 result carries its own rounding, 1.7e-3.
    if case["kind"] in ("self", "cross", "nag") and case["dtype"] == "bf16":
        return {"rel": 7e-3}
    return {"rel": {"mlp": 8e-4, "cross_kv": 1.2e-3}.get(case["kind"], 2e-3)}
