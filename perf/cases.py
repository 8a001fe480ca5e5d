"""What a user of this framework has it do, as cases that can be timed and compared.

``listed()`` names the cases, ``draw(rng)`` makes further ones over the same ranges, ``prepare`` builds what the
user's program holds before the call, ``run`` is one pass through the public entry points.

Kinds and the ranges they stand for:

* ``flux_attn``   joint attention of a Flux layer from its fused q/k/v projection (per-head RMSNorm, per-token rotary
                  table): 256 to 8192 image tokens, 77 to 512 text tokens, batch 1 or 2
* ``wan_attn``    self-attention of a Wan layer from its fused projection (full-width RMSNorm, three-axis rotary):
                  12 or 40 heads, one latent frame at 240p to 21 frames at 720p
* ``attn``        the attention backend called with q / k / v: cross-attention to the text tokens and plain calls of
                  ragged lengths, bf16 and fp16, with and without the log-sum-exp
* ``ring``        one rank's share of ring attention: every source block attended with its log-sum-exp and folded into
                  an ``AttentionState``
* ``q8``          the 8-bit backend (INT8 scores, E4M3 values)
* ``flux_blocks`` one double-stream and two single-stream Flux blocks (the model's 19 : 38)
* ``wan_block``   one Wan block: self-attention, cross-attention to the text, feed-forward
* ``qwen_block``  one Qwen-Image MMDiT block
* ``cfg``         the classifier-free-guidance combine that ends every denoising step
"""

from __future__ import annotations

import math

import torch

from chitudiffusion_b200 import B200AttnBackend, ops
from chitudiffusion_b200.dit import WanBlock
from chitudiffusion_b200.flux_dit import FluxDoubleBlock, FluxSingleBlock
from chitudiffusion_b200.pre_attention import JointPreAttention, WanPreAttention, axis_rope_table
from chitudiffusion_b200.qwen import B200QwenAttnProcessor, QwenDoubleBlock
from chitudiffusion_b200.state import AttentionState

HEAD_DIM = 128
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # the classifier-free-guidance combine of a 1328 x 1328 Qwen-Image step, rescaled to the conditional norm:
        # the smallest call, one launch
        {"name": "cfg-qwen-1328", "kind": "cfg", "batch": 1, "rows": 6889, "channels": 64, "dtype": "bf16",
         "rescale": True},
        # a 256 x 256 Flux preview: 16 x 16 image tokens behind 512 text tokens, latency of one layer
        {"name": "flux-attn-256px", "kind": "flux_attn", "batch": 1, "img_h": 16, "img_w": 16, "txt": 512, "heads": 24},
        # Flux at 1024 x 1024, the layer that the benchmark's step consists of
        {"name": "flux-attn-1024px", "kind": "flux_attn", "batch": 1, "img_h": 64, "img_w": 64, "txt": 512, "heads": 24},
        # Wan2.1-1.3B, 480p, 17 frames
        {"name": "wan1.3b-attn-480p-17f", "kind": "wan_attn", "batch": 1, "grid_f": 5, "grid_h": 30, "grid_w": 52,
         "heads": 12},
        # Wan2.1-14B, 720p, 81 frames: the largest
        {"name": "wan14b-attn-720p-81f", "kind": "wan_attn", "batch": 1, "grid_f": 21, "grid_h": 45, "grid_w": 80,
         "heads": 40},
        # Wan2.1-1.3B cross-attention: every video token against 512 text tokens
        {"name": "wan1.3b-cross-480p-81f", "kind": "attn", "batch": 1, "sq": 32760, "sk": 512, "heads": 12,
         "dtype": "bf16", "lse": False},
        # a plain backend call in fp16 with ragged lengths, batch 2 (both guidance branches) and the log-sum-exp
        {"name": "attn-fp16-ragged-b2", "kind": "attn", "batch": 2, "sq": 1037, "sk": 1331, "heads": 24,
         "dtype": "fp16", "lse": True},
        # ring attention of Wan2.1-1.3B at 480p over four ranks: one rank's queries, four key blocks, merged partials
        {"name": "wan1.3b-ring4-480p-81f", "kind": "ring", "batch": 1, "rows": 8190, "blocks": 4, "heads": 12},
        # Qwen-Image at 1328 x 1328 with the 8-bit backend
        {"name": "q8-qwen-1328", "kind": "q8", "batch": 1, "seq": 7145, "heads": 24},
        # Flux blocks at 1024 x 1024: a double-stream and two single-stream blocks
        {"name": "flux-blocks-1024px", "kind": "flux_blocks", "batch": 1, "img_h": 64, "img_w": 64, "txt": 512,
         "dim": 3072, "heads": 24},
        # a Wan2.1-1.3B block at 480p, 81 frames
        {"name": "wan1.3b-block-480p-81f", "kind": "wan_block", "batch": 1, "grid_f": 21, "grid_h": 30, "grid_w": 52,
         "dim": 1536, "ffn": 8960, "heads": 12, "txt": 512},
        # a Qwen-Image block at 1328 x 1328 with a prompt of 217 tokens
        {"name": "qwen-block-1328", "kind": "qwen_block", "batch": 1, "img_h": 83, "img_w": 83, "txt": 217,
         "dim": 3072, "heads": 24},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _text_tokens(rng):
    return rng.choice([77, 256, 512, rng.randint(77, 512)])


def _wan_grid(rng, max_tokens):
    """Latent grid of a clip: 1 to 21 latent frames of 240p to 720p."""
    while True:
        g = {"grid_f": _log_int(rng, 1, 21), "grid_h": rng.randint(15, 45), "grid_w": rng.randint(26, 80)}
        if g["grid_f"] * g["grid_h"] * g["grid_w"] <= max_tokens:
            return g


def _image_grid(rng, max_tokens):
    tokens = _log_int(rng, 256, max_tokens)
    h = max(8, int(round(math.sqrt(tokens) * rng.uniform(0.6, 1.4))))
    return {"img_h": h, "img_w": max(8, tokens // h)}


def draw(rng):
    kind = rng.choice(["flux_attn", "flux_attn", "wan_attn", "wan_attn", "attn", "attn", "ring", "q8", "flux_blocks",
                       "wan_block", "qwen_block", "cfg"])
    if kind == "flux_attn":
        return {"kind": kind, "batch": rng.choice([1, 1, 2]), **_image_grid(rng, 8192), "txt": _text_tokens(rng),
                "heads": 24}
    if kind == "wan_attn":
        heads = rng.choice([12, 40])
        return {"kind": kind, "batch": rng.choice([1, 1, 2]), **_wan_grid(rng, 48000 if heads == 12 else 32000),
                "heads": heads}
    if kind == "attn":
        sq = _log_int(rng, 128, 33000)
        sk = rng.choice([rng.randint(64, 512), _log_int(rng, 128, 12000)])
        return {"kind": kind, "batch": rng.choice([1, 2]), "sq": sq, "sk": sk, "heads": rng.choice([5, 12, 24, 40]),
                "dtype": rng.choice(["bf16", "bf16", "fp16"]), "lse": rng.choice([True, False])}
    if kind == "ring":
        return {"kind": kind, "batch": 1, "rows": _log_int(rng, 512, 9000), "blocks": rng.choice([2, 4, 8]),
                "heads": rng.choice([12, 24])}
    if kind == "q8":
        return {"kind": kind, "batch": rng.choice([1, 1, 2]), "seq": _log_int(rng, 768, 16000), "heads": rng.choice([12, 24])}
    if kind == "flux_blocks":
        return {"kind": kind, "batch": rng.choice([1, 1, 2]), **_image_grid(rng, 4400), "txt": _text_tokens(rng),
                "dim": 3072, "heads": 24}
    if kind == "wan_block":
        return {"kind": kind, "batch": rng.choice([1, 1, 2]), **_wan_grid(rng, 33000), "dim": 1536, "ffn": 8960,
                "heads": 12, "txt": _text_tokens(rng)}
    if kind == "qwen_block":
        return {"kind": kind, "batch": rng.choice([1, 1, 2]), **_image_grid(rng, 7000), "txt": _text_tokens(rng),
                "dim": 3072, "heads": 24}
    # guidance: token rows of an image model, or [frames * rows, columns] of a video latent
    if rng.random() < 0.5:
        return {"kind": "cfg", "batch": rng.choice([1, 2]), "rows": _log_int(rng, 1000, 16000), "channels": 64,
                "dtype": "bf16", "rescale": rng.choice([True, False])}
    return {"kind": "cfg", "batch": rng.choice([1, 2]), "rows": 16 * rng.randint(1, 21) * rng.randint(30, 90),
            "channels": 2 * rng.randint(26, 80), "dtype": rng.choice(["fp32", "bf16"]), "rescale": False}


# ------------------------------------------------------------------------------------------- inputs
def _gen(seed, device):
    return torch.Generator(device=device).manual_seed(int(seed))


def _randn(shape, gen, dtype, scale=1.0):
    x = torch.randn(shape, generator=gen, device=gen.device)
    return (x * scale if scale != 1.0 else x).to(dtype)


def _image_ids(n_txt, h, w):
    """Position ids of the joint [text, image] sequence: text at the origin, image tokens at (row, column)."""
    ids = torch.zeros(n_txt + h * w, 3)
    ids[n_txt:, 1] = torch.arange(h).repeat_interleave(w)
    ids[n_txt:, 2] = torch.arange(w).repeat(h)
    return ids


def _complex_freqs(ids, axes_dims):
    t = axis_rope_table(ids, axes_dims)
    return torch.complex(t[..., 0], t[..., 1])


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = _gen(seed, dev)
    kind, B = case["kind"], case["batch"]
    if kind == "cfg":
        shape = (B, case["rows"], case["channels"])
        cond = _randn(shape, gen, torch.float32)
        uncond = cond + 0.3 * _randn(shape, gen, torch.float32)  # the two branches are close
        dt = DTYPES[case["dtype"]]
        return {"case": case, "cond": cond.to(dt), "uncond": uncond.to(dt)}
    H = case["heads"]
    C = H * HEAD_DIM
    if kind == "attn":
        dt = DTYPES[case["dtype"]]
        q = _randn((B, case["sq"], H, HEAD_DIM), gen, dt)
        k = _randn((B, case["sk"], H, HEAD_DIM), gen, dt)
        v = _randn((B, case["sk"], H, HEAD_DIM), gen, dt)
        return {"case": case, "attn": B200AttnBackend("b200"), "q": q, "k": k, "v": v}
    if kind == "ring":
        shape = (B, case["rows"], H, HEAD_DIM)
        blocks = [(_randn(shape, gen, torch.bfloat16), _randn(shape, gen, torch.bfloat16))
                  for _ in range(case["blocks"])]
        return {"case": case, "attn": B200AttnBackend("b200"), "q": _randn(shape, gen, torch.bfloat16), "blocks": blocks}
    if kind == "q8":
        shape = (B, case["seq"], H, HEAD_DIM)
        q, k, v = (_randn(shape, gen, torch.bfloat16) for _ in range(3))
        # keys carry a per-channel offset, which the 8-bit path takes out before it quantises them
        k = (k.float() + _randn((1, 1, H, HEAD_DIM), gen, torch.float32)).to(torch.bfloat16)
        return {"case": case, "attn": B200AttnBackend("b200_q8"), "q": q, "k": k, "v": v}
    if kind == "flux_attn":
        S = case["txt"] + case["img_h"] * case["img_w"]
        table = axis_rope_table(_image_ids(case["txt"], case["img_h"], case["img_w"]), (16, 56, 56), device=dev)
        return {"case": case, "attn": B200AttnBackend("b200"), "pre": JointPreAttention(H, HEAD_DIM, table),
                "qkv": _randn((B, S, 3 * C), gen, torch.bfloat16),
                "wq": 1.0 + _randn((HEAD_DIM,), gen, torch.float32, 0.1),
                "wk": 1.0 + _randn((HEAD_DIM,), gen, torch.float32, 0.1)}
    if kind == "wan_attn":
        grid = (case["grid_f"], case["grid_h"], case["grid_w"])
        S = grid[0] * grid[1] * grid[2]
        return {"case": case, "attn": B200AttnBackend("b200"), "pre": WanPreAttention(H, HEAD_DIM, device=dev),
                "grid": grid, "qkv": _randn((B, S, 3 * C), gen, torch.bfloat16),
                "wq": 1.0 + _randn((C,), gen, torch.float32, 0.1), "wk": 1.0 + _randn((C,), gen, torch.float32, 0.1)}
    dim = case["dim"]
    if kind == "flux_blocks":
        n_img = case["img_h"] * case["img_w"]
        table = axis_rope_table(_image_ids(case["txt"], case["img_h"], case["img_w"]), (16, 56, 56), device=dev)
        return {"case": case, "attn": B200AttnBackend("b200"), "table": table,
                "double": [FluxDoubleBlock.random_init(dim, H, dev, seed=int(seed) % 100003)],
                "single": [FluxSingleBlock.random_init(dim, H, dev, seed=int(seed) % 100003 + 1 + i) for i in range(2)],
                "img": _randn((B, n_img, dim), gen, torch.bfloat16), "txt": _randn((B, case["txt"], dim), gen, torch.bfloat16),
                "temb": _randn((B, dim), gen, torch.bfloat16)}
    if kind == "wan_block":
        grid = (case["grid_f"], case["grid_h"], case["grid_w"])
        S = grid[0] * grid[1] * grid[2]
        return {"case": case, "attn": B200AttnBackend("b200"), "pre": WanPreAttention(H, dim // H, device=dev), "grid": grid,
                "block": WanBlock.random_init(dim, case["ffn"], H, dev, seed=int(seed) % 100003),
                "x": _randn((B, S, dim), gen, torch.float32), "e": _randn((B, 6, dim), gen, torch.float32, 0.3),
                "context": _randn((B, case["txt"], dim), gen, torch.bfloat16)}
    n_img = case["img_h"] * case["img_w"]
    ids = _image_ids(0, case["img_h"], case["img_w"])
    txt_ids = torch.arange(case["txt"]).float().add(max(case["img_h"], case["img_w"]))[:, None].expand(-1, 3)
    rotary = (_complex_freqs(ids, (16, 56, 56)).to(dev), _complex_freqs(txt_ids, (16, 56, 56)).to(dev))
    return {"case": case, "block": QwenDoubleBlock.random_init(dim, H, dev, seed=int(seed) % 100003),
            "processor": B200QwenAttnProcessor(B200AttnBackend("b200")), "rotary": rotary,
            "img": _randn((B, n_img, dim), gen, torch.bfloat16), "txt": _randn((B, case["txt"], dim), gen, torch.bfloat16),
            "temb": _randn((B, dim), gen, torch.bfloat16)}


# --------------------------------------------------------------------------------------------- pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "cfg":
        return ops.cfg_combine(state["cond"], state["uncond"], 4.0, rescale=case["rescale"])
    if kind == "attn":
        out, lse, _ = state["attn"](state["q"], state["k"], state["v"], return_attn_probs=case["lse"])
        return (out, lse) if case["lse"] else out
    if kind == "q8":
        return state["attn"](state["q"], state["k"], state["v"])[0]
    if kind == "ring":
        acc = AttentionState()
        for k, v in state["blocks"]:
            out, lse, _ = state["attn"](state["q"], k, v, return_attn_probs=True)
            acc.update(out, lse)
        return acc.out, acc.lse
    if kind in ("flux_attn", "wan_attn"):
        qkv, pre = state["qkv"], state["pre"]
        C = qkv.shape[2] // 3
        args = pre.batch_args(qkv.shape[1], state["grid"]) if kind == "wan_attn" else pre.batch_args(qkv.shape[1])
        return state["attn"].attention_from_projections(
            pre.jobs(qkv[..., :C], qkv[..., C:2 * C], state["wq"], state["wk"]), qkv[..., 2 * C:], **args)
    # the residual streams are updated in place: a denoising step starts from a fresh embedding of its latents
    if kind == "flux_blocks":
        img, txt = state["img"].clone(), state["txt"].clone()
        for blk in state["double"]:
            txt, img = blk(img, txt, state["temb"], state["table"], state["attn"])
        x = torch.cat([txt, img], dim=1)
        for blk in state["single"]:
            x = blk(x, state["temb"], state["table"], state["attn"])
        return x
    if kind == "wan_block":
        return state["block"](state["x"].clone(), state["e"], state["grid"], state["context"], state["attn"], state["pre"])
    return state["block"](state["img"].clone(), state["txt"].clone(), state["temb"], state["rotary"], state["processor"])


# ------------------------------------------------------------------------------- work and tolerance
def work(case):
    kind, B = case["kind"], case["batch"]
    if kind == "cfg":
        n = B * case["rows"] * case["channels"]
        return {"bytes": 3 * n * (4 if case["dtype"] == "fp32" else 2), "flops": 3 * n}
    H = case["heads"]
    C = H * HEAD_DIM
    if kind == "attn":
        return {"bytes": 2 * B * C * (2 * case["sq"] + 2 * case["sk"]) + (4 * B * H * case["sq"] if case["lse"] else 0),
                "flops": 4 * B * case["sq"] * case["sk"] * C}
    if kind == "ring":
        n = case["rows"]
        return {"bytes": 2 * B * C * n * (1 + 2 * case["blocks"]) + 4 * B * n * (C + H),
                "flops": 4 * B * n * n * case["blocks"] * C}
    if kind == "q8":
        n = case["seq"]
        return {"bytes": 8 * B * n * C, "flops": 4 * B * n * n * C}
    if kind in ("flux_attn", "wan_attn"):
        n = (case["txt"] + case["img_h"] * case["img_w"] if kind == "flux_attn"
             else case["grid_f"] * case["grid_h"] * case["grid_w"])
        return {"bytes": 8 * B * n * C, "flops": 4 * B * n * n * C}
    dim = case["dim"]
    if kind == "flux_blocks":
        n_img, n_txt = case["img_h"] * case["img_w"], case["txt"]
        n = n_img + n_txt
        attn = 3 * 4 * B * n * n * dim
        gemm = 2 * B * dim * dim * (12 * n + 2 * 12 * n) + 2 * B * dim * dim * (12 + 2 * 3)
        weights = 2 * dim * dim * (2 * 18 + 2 * 15)
        return {"bytes": weights + 4 * B * n * dim, "flops": attn + gemm}
    if kind == "wan_block":
        n, t, f = case["grid_f"] * case["grid_h"] * case["grid_w"], case["txt"], case["ffn"]
        attn = 4 * B * n * (n + t) * dim
        gemm = 2 * B * dim * (n * (6 * dim + 2 * f) + t * 2 * dim)
        return {"bytes": 2 * dim * (8 * dim + 2 * f) + 8 * B * n * dim + 2 * B * t * dim, "flops": attn + gemm}
    n_img, n_txt = case["img_h"] * case["img_w"], case["txt"]
    n = n_img + n_txt
    return {"bytes": 2 * dim * dim * 36 + 4 * B * n * dim, "flops": 4 * B * n * n * dim + 2 * B * dim * dim * (12 * n + 12)}


# About four times the relative error against the same path in 64 bits, measured at reduced sizes of each kind
# (bf16 attention 2.3e-3, with the norm + rotary pass in front 3.4e-3, fp16 attention 2.9e-4, Flux blocks 5.9e-3, Qwen
# block 4.4e-3, Wan block with its fp32 stream 1.0e-3, guidance 1.7e-3 in bf16).  8 bits: 4.0e-2, of which the E4M3 roundings of
# the probabilities (half of its square) depend on where the running maximum stood when they were formed, so two
# correct implementations differ by up to about that much.
REL = {"attn": 1e-2, "ring": 1e-2, "q8": 6e-2, "flux_attn": 1.3e-2, "wan_attn": 1.3e-2, "flux_blocks": 2.3e-2,
       "wan_block": 4e-3, "qwen_block": 1.7e-2, "cfg": 6e-3}


def tolerance(case):
    if case.get("dtype") == "fp16":
        return {"rel": 1.2e-3}
    if case.get("dtype") == "fp32":
        return {"rel": 1e-5}
    return {"rel": REL[case["kind"]]}
