"""The work that programs on this library have it do, as cases that can be timed and compared.

Four families, each entered the way a program enters it:

  attention   `fmha_forward_kernel` on caller-owned buffers: prefill (causal, or with an additive bias),
              the self- and cross-attention of image models in [B, S, N, H] storage and fp16, and
              decode against a [B, T, N, H] cache with one to sixteen new rows per sequence
  training    the same forward with its log-sum-exp rows kept, then `fmha_backward_kernel`
  gemm        `gemm` with an epilogue (token counts are ragged, weights are not), and `gemm_fp8`
              on operands quantised per tensor
  layers      `gptj_layer_prefill` and `gemma_decode_step`: a decoder layer's whole chain of calls

Attention inputs are N(0, 1), weights N(0, 0.02), as the benchmark configurations state.
"""
import importlib
import math

import torch

PACKAGE = "intel-extension-for-openxla_b200"
ixk = importlib.import_module(PACKAGE)
layers = importlib.import_module(PACKAGE + ".layers")

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "e4m3": torch.float8_e4m3fn, "e5m2": torch.float8_e5m2}

# Decoder layer widths: the GPT-J-6B-shaped block and the Gemma-7B-shaped block of the benchmark.
GPTJ = {"hidden": 4096, "heads": 16, "head_dim": 256, "rotary": 64, "ffn": 16384}
GEMMA = {"hidden": 3072, "heads": 16, "head_dim": 256, "ffn": 24576}


def _attention(name, B, N, F, T, H, dtype="bf16", causal=False, bias="none", storage="bnsh", family="attention"):
    return {"name": name, "family": family, "B": B, "N": N, "F": F, "T": T, "H": H, "dtype": dtype, "causal": causal,
            "bias": bias, "storage": storage}


def listed():
    return [
        # causal prefill of a 128-wide-head model: the headline configuration
        _attention("prefill_causal_h128", 8, 16, 2048, 2048, 128, causal=True),
        # the same sizes under a per-batch additive bias (relative positions, padding masks)
        _attention("prefill_bias_h128", 8, 16, 2048, 2048, 128, bias="batch"),
        # self-attention of a diffusion model's 64 x 64 latent, two images (classifier-free guidance)
        _attention("image_self_h64", 2, 10, 4096, 4096, 64, dtype="fp16", storage="bsnh"),
        # cross-attention of the same family to a 77-token prompt: a small call, made dozens of times a step
        _attention("image_text_h64", 2, 20, 1024, 77, 64, dtype="fp16", storage="bsnh"),
        # four drafted tokens per sequence checked against a ragged cache (speculative decoding)
        _attention("decode_4rows_h256", 32, 16, 4, 3001, 256, storage="bsnh"),
        # attention of a training step, forward and backward, at the headline sizes
        _attention("train_causal_h128", 8, 16, 2048, 2048, 128, causal=True, family="training"),
        # and with the 256-wide heads of both decoder layers (fine-tuning)
        _attention("train_causal_h256", 4, 16, 2048, 2048, 256, causal=True, storage="bsnh", family="training"),
        # an MLP up-projection with its fused epilogue for a batch of prompts of uneven length
        {"name": "gemm_bias_gelu_ragged", "family": "gemm", "M": 1371, "N": 16384, "K": 4096, "dtype": "bf16",
         "epilogue": "BIAS_GELU", "weight": "row"},
        # the scaled fp8 product of the fp8 configuration
        {"name": "gemm_fp8", "family": "gemm_fp8", "M": 16384, "N": 8192, "K": 8192, "a": "e4m3", "b": "e4m3"},
        # a whole decoder layer on four prompts of 2048 tokens
        {"name": "gptj_prefill", "family": "gptj", "B": 4, "S": 2048},
        # one token for each of 64 sequences, caches nearly full: the serving configuration
        {"name": "gemma_decode_batch", "family": "gemma", "B": 64, "capacity": 4096, "position": 4095},
        # one token for a single user
        {"name": "gemma_decode_single", "family": "gemma", "B": 1, "capacity": 2048, "position": 1000},
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    """One more case of the same ranges; no drawn case costs more than the largest listed one."""
    kind = rng.choice(["prefill", "prefill", "image", "decode", "training", "training", "gemm", "gemm", "gemm_fp8", "gptj", "gemma"])
    if kind == "prefill":
        H = rng.choice([40, 64, 80, 128, 128, 128, 160, 256])
        S = _log_int(rng, 17, 4096)
        N = rng.choice([4, 8, 12, 16])
        B = max(1, min(_log_int(rng, 1, 16), int(6e8 / (N * S * max(S, 128)))))
        causal = rng.random() < 0.6
        bias = "none" if causal and rng.random() < 0.7 else rng.choice(["none", "batch", "head"])
        if B * (N if bias == "head" else 1) * S * S > 3e8:
            bias = "none"
        c = _attention("", B, N, S, S, H, rng.choice(["bf16", "bf16", "fp16"]), causal, bias, rng.choice(["bnsh", "bsnh"]))
    elif kind == "image":
        # latents of side 8 to 96, alone or with their text
        side, B = _log_int(rng, 8, 96), rng.choice([1, 2, 4])
        N, H = rng.choice([(5, 64), (10, 64), (20, 64), (8, 40), (8, 80), (8, 160)])
        T = rng.choice([77, side * side]) if B * N * side ** 4 < 1e9 else 77
        c = _attention("", B, N, side * side, T, H, rng.choice(["bf16", "fp16"]), storage="bsnh")
    elif kind == "decode":
        B, N, H = _log_int(rng, 1, 64), rng.choice([8, 16]), rng.choice([64, 128, 256])
        T = _log_int(rng, 33, 4096)
        c = _attention("", B, N, rng.choice([1, 1, 2, 3, 4, 5, 8, 16]), T, H, rng.choice(["bf16", "bf16", "fp16"]), storage="bsnh")
    elif kind == "training":
        H = rng.choice([64, 128, 128, 256, 256])
        S = _log_int(rng, 65, 2048)
        N = rng.choice([8, 12, 16])
        B = max(1, min(_log_int(rng, 1, 16), int(3.4e10 / (N * S * max(S, 256) * H))))
        c = _attention("", B, N, S, S, H, rng.choice(["bf16", "bf16", "fp16"]), rng.random() < 0.7,
                       storage=rng.choice(["bnsh", "bsnh"]), family="training")
    elif kind == "gemm":
        N, K = _log_int(rng, 256, 16384, 8), _log_int(rng, 256, 16384, 8)
        M = min(_log_int(rng, 1, 8192), max(1, int(5.5e11 / (N * K))))
        c = {"family": "gemm", "M": M, "N": N, "K": K, "dtype": rng.choice(["bf16", "bf16", "fp16"]),
             "epilogue": rng.choice(["DEFAULT", "BIAS", "GELU", "BIAS_GELU", "BIAS_RELU"]), "weight": rng.choice(["row", "row", "col"])}
    elif kind == "gemm_fp8":
        N, K = _log_int(rng, 512, 8192, 16), _log_int(rng, 512, 8192, 16)
        M = _log_int(rng, 16, 16384)
        c = {"family": "gemm_fp8", "M": M, "N": N, "K": K, "a": "e4m3", "b": rng.choice(["e4m3", "e5m2"])}
    elif kind == "gptj":
        S = _log_int(rng, 16, 2048)
        c = {"family": "gptj", "B": max(1, min(_log_int(rng, 1, 8), 8192 // S)), "S": S}
    else:
        capacity = _log_int(rng, 128, 4096)
        c = {"family": "gemma", "B": _log_int(rng, 1, 64), "capacity": capacity, "position": rng.randrange(capacity // 2, capacity)}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------------------------- preparation

def _randn(g, *shape, dtype=torch.bfloat16, scale=1.0):
    t = torch.randn(*shape, generator=g, device="cuda", dtype=dtype)
    return t.mul_(scale) if scale != 1.0 else t


def _heads(g, B, N, S, H, dtype, storage):
    """[B, N, S, H] view of a tensor in the given storage order."""
    if storage == "bsnh":
        return _randn(g, B, S, N, H, dtype=dtype).permute(0, 2, 1, 3)
    return _randn(g, B, N, S, H, dtype=dtype)


def _workspace(nbytes):
    return torch.empty(max(int(nbytes), 16), dtype=torch.uint8, device="cuda")


def prepare(case, seed):
    """What the program holds when it makes the call: inputs, weights, output buffers, scratch."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    c = case
    if c["family"] in ("attention", "training"):
        B, N, F, T, H, dt, st = c["B"], c["N"], c["F"], c["T"], c["H"], DTYPES[c["dtype"]], c["storage"]
        s = {"case": c, "q": _heads(g, B, N, F, H, dt, st), "k": _heads(g, B, N, T, H, dt, st), "v": _heads(g, B, N, T, H, dt, st),
             "bias": None, "lse": None, "scale": H ** -0.5}
        s["out"] = torch.empty_like(s["q"])
        if c["bias"] != "none":
            s["bias"] = _randn(g, B, N if c["bias"] == "head" else 1, F, T, dtype=dt)
        s["workspace"] = _workspace(ixk.fmha_workspace_bytes(s["q"], s["k"], s["v"], s["bias"], s["out"], s["scale"], c["causal"]))
        if c["family"] == "training":
            s["lse"] = torch.empty(B, N, F, dtype=torch.float32, device="cuda")
            s["grad_out"] = _heads(g, B, N, F, H, dt, st)
            for name, like in (("dq", "q"), ("dk", "k"), ("dv", "v")):
                s[name] = torch.empty_like(s[like])
            s["bwd_workspace"] = _workspace(ixk.fmha_backward_workspace_bytes(
                s["q"], s["k"], s["v"], s["out"], s["bias"], s["grad_out"], s["dq"], s["dk"], s["dv"], s["scale"], c["causal"]))
        return s
    if c["family"] == "gemm":
        dt = DTYPES[c["dtype"]]
        w = (_randn(g, c["N"], c["K"], dtype=dt, scale=0.02).t() if c["weight"] == "col"
             else _randn(g, c["K"], c["N"], dtype=dt, scale=0.02))
        s = {"case": c, "x": _randn(g, c["M"], c["K"], dtype=dt), "w": w,
             "bias": _randn(g, c["N"], dtype=dt, scale=0.02) if "BIAS" in c["epilogue"] else None}
        s["workspace"] = _workspace(ixk.gemm_workspace_bytes(s["x"], w))
        return s
    if c["family"] == "gemm_fp8":
        s = {"case": c}
        for name, rows, cols in (("a", c["M"], c["K"]), ("b", c["K"], c["N"])):
            q, scale = ixk.quantize_fp8(_randn(g, rows, cols, dtype=torch.float32), DTYPES[c[name]])
            s[name], s["inv_" + name] = q, 1.0 / scale
        return s
    if c["family"] == "gptj":
        h, f, hd = GPTJ["hidden"], GPTJ["ffn"], GPTJ["heads"] * GPTJ["head_dim"]
        r = lambda *shape: _randn(g, *shape, scale=0.02)  # noqa: E731
        w = layers.GptJLayerWeights(wqkv=r(h, 3 * hd), wo=r(hd, h), w1=r(h, f), b1=r(f), w2=r(f, h), b2=r(h),
                                    heads_local=GPTJ["heads"], head_dim=GPTJ["head_dim"], rotary_dim=GPTJ["rotary"])
        return {"case": c, "x": _randn(g, c["B"], c["S"], h), "w": w, "ops": layers.KernelOps(ixk, gemm_workspace=_workspace(32 << 20)),
                "rope": layers.rotary_tables(torch.arange(c["S"], device="cuda"), GPTJ["rotary"])}
    h, f, N, H = GEMMA["hidden"], GEMMA["ffn"], GEMMA["heads"], GEMMA["head_dim"]
    r = lambda *shape: _randn(g, *shape, scale=0.02)  # noqa: E731
    w = layers.GemmaLayerWeights(wqkv=r(h, 3 * N * H), wo=r(N * H, h), wgateup=r(h, 2 * f), wdown=r(f, h), heads_local=N, head_dim=H,
                                 norm_attn=r(h), norm_mlp=r(h))
    B, T = c["B"], c["capacity"]
    return {"case": c, "x": _randn(g, B, 1, h), "w": w, "k_cache": _randn(g, B, T, N, H), "v_cache": _randn(g, B, T, N, H),
            "ops": layers.KernelOps(ixk, gemm_workspace=_workspace(32 << 20)), "workspace": _workspace(8 << 20),
            "rope": layers.rotary_tables(torch.tensor([c["position"]], device="cuda"), H)}


# ------------------------------------------------------------------------------------- one pass

def run(state):
    s, c = state, state["case"]
    if c["family"] == "attention":
        ixk.fmha_forward_kernel(None, s["q"], s["k"], s["v"], s["bias"], None, 0.0, s["out"], None, s["scale"], False,
                                causal=c["causal"], workspace=s["workspace"])
        return s["out"]
    if c["family"] == "training":
        ixk.fmha_forward_kernel(None, s["q"], s["k"], s["v"], s["bias"], None, 0.0, s["out"], s["lse"], s["scale"], True,
                                causal=c["causal"], workspace=s["workspace"])
        ixk.fmha_backward_kernel(None, s["q"], s["k"], s["v"], s["out"], s["bias"], s["grad_out"], s["lse"], s["dq"], s["dk"],
                                 s["dv"], s["scale"], causal=c["causal"], workspace=s["bwd_workspace"])
        return {name: s[name] for name in ("out", "lse", "dq", "dk", "dv")}
    if c["family"] == "gemm":
        return ixk.gemm(s["x"], s["w"], bias=s["bias"], epilogue=c["epilogue"], workspace=s["workspace"])
    if c["family"] == "gemm_fp8":
        return ixk.gemm_fp8(s["a"], s["b"], s["inv_a"], s["inv_b"])
    if c["family"] == "gptj":
        return layers.gptj_layer_prefill(s["x"], s["w"], s["ops"], rope=s["rope"])
    y = layers.gemma_decode_step(s["x"], s["w"], s["k_cache"], s["v_cache"], c["position"], s["ops"], workspace=s["workspace"],
                                 rope=s["rope"])
    return {"y": y, "k_cache": s["k_cache"], "v_cache": s["v_cache"]}


# ------------------------------------------------------------------------------------- what it takes

def _pairs(c):
    """(query, key) pairs that the mask leaves."""
    F, T = c["F"], c["T"]
    if not c["causal"]:
        return F * T
    full = min(F, T)
    return full * (full + 1) // 2 + (F - full) * T


def work(case):
    c = case
    if c["family"] in ("attention", "training"):
        B, N, F, T, H = c["B"], c["N"], c["F"], c["T"], c["H"]
        q, kv = 2.0 * B * N * F * H, 2.0 * B * N * T * H
        nbytes, flops = 2 * q + 2 * kv, 4.0 * B * N * _pairs(c) * H
        if c["bias"] != "none":
            nbytes += 2.0 * B * (N if c["bias"] == "head" else 1) * F * T
        if c["family"] == "training":  # + grad_out in, dq, dk and dv out; five products behind the forward's two
            nbytes += 2 * q + 2 * kv + 4.0 * B * N * F
            flops *= 3.5
        return {"bytes": nbytes, "flops": flops}
    if c["family"] == "gemm":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": 2.0 * (M * K + K * N + M * N), "flops": 2.0 * M * N * K}
    if c["family"] == "gemm_fp8":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": 1.0 * (M * K + K * N) + 2.0 * M * N, "flops": 2.0 * M * N * K}
    if c["family"] == "gptj":
        m, h, f, hd = c["B"] * c["S"], GPTJ["hidden"], GPTJ["ffn"], GPTJ["heads"] * GPTJ["head_dim"]
        weights = h * 3 * hd + hd * h + 2 * h * f
        return {"bytes": 2.0 * (weights + 2 * m * h),
                "flops": layers.gptj_layer_flops(c["B"], c["S"], h, GPTJ["heads"], GPTJ["head_dim"], f)}
    h, f, hd, B, T = GEMMA["hidden"], GEMMA["ffn"], GEMMA["heads"] * GEMMA["head_dim"], c["B"], c["position"] + 1
    weights = h * 3 * hd + hd * h + 3 * h * f
    return {"bytes": layers.gemma_decode_bytes(B, T, h, GEMMA["heads"], GEMMA["head_dim"], f),
            "flops": 2.0 * B * weights + 4.0 * B * T * hd}


def tolerance(case):
    """About four times the distance (2-norm) of each family's results from the same formulas in 64-bit arithmetic:
    bf16 attention 2.4e-3 and its gradients 3.1e-3, bf16 and fp8 products 1.7e-3 (one rounding to bf16), the GPT-J
    block 3.9e-3, the Gemma step 4.9e-3; fp16, with three more bits, 3e-4 (gradients 3.9e-4)."""
    if case["family"] in ("attention", "training"):
        return {"rel": 1.2e-2 if case["dtype"] == "bf16" else 1.5e-3}
    if case["family"] in ("gemm", "gemm_fp8"):
        return {"rel": 1e-3 if case.get("dtype") == "fp16" else 7e-3}
    return {"rel": 1.5e-2 if case["family"] == "gptj" else 2e-2}
