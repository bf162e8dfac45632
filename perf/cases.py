"""The performance cases of sageattention_b200: attention calls as models make them, from one short head pair to a
119 056-token video clip, through the public entry points (`sageattn3`, `sageattn`, `sageattn_varlen`).

A case is a dict of plain values:
  entry    "dense" (sageattn3), "lse" (sageattn with return_lse) or "varlen" (sageattn_varlen)
  B, Hq, Hkv, Nq, Nk, D, dtype ("bf16" / "fp16"), causal, layout ("HND" / "NHD")
  block_mean   Q smoothed per 128-row block (True) or by one mean per head (False)
  scale        softmax scale relative to D ** -0.5 (1.0: the default, not passed)
  k_dist       what makes K worth smoothing: "offset" (a mean per channel), "outlier" (four channels twice as large) or
               "rope" (rotated by position, base 500 000, as language models do; Q too)
  len_min, len_seed    varlen only: lengths spread over [len_min, Nq], drawn from len_seed, the longest being Nq
"""
import math
import random

import torch

from sageattention_b200 import sageattn, sageattn3, sageattn_varlen

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _case(B, Hq, Hkv, Nq, Nk, D, dtype="bf16", causal=False, layout="HND", k_dist="offset", entry="dense", block_mean=True,
          scale=1.0, **more):
    return dict(entry=entry, B=B, Hq=Hq, Hkv=Hkv, Nq=Nq, Nk=Nk, D=D, dtype=dtype, causal=causal, layout=layout,
                k_dist=k_dist, block_mean=block_mean, scale=scale, **more)


def listed():
    named = [
        # A thousand tokens of two heads: the smallest self-attention in use; all launches and latency.
        ("short_1k", _case(1, 2, 2, 1024, 1024, 128)),
        # One step of token generation with SDPA patched: a new token of eight sequences against 8 192 cached keys.
        ("decode_8k", _case(8, 32, 8, 1, 8192, 128, causal=True, layout="NHD", k_dist="rope")),
        # A later chunk of a long prompt: 1 000 new tokens against 9 192 keys, mask aligned at the bottom right.
        ("chunk_1000_of_9k", _case(1, 32, 8, 1000, 9192, 128, causal=True, layout="NHD", k_dist="rope")),
        # The prompt of one request, of no round length, as a serving engine prefills it.
        ("prompt_3001", _case(1, 32, 8, 3001, 3001, 128, causal=True, layout="NHD", k_dist="rope")),
        # Cross-attention of a video transformer: every video token against 226 text tokens.
        ("cross_text_226", _case(2, 48, 48, 17550, 226, 64, layout="NHD")),
        # One block of an image diffusion transformer, 4 096 image + 154 text tokens, with guidance (batch 2).
        ("image_4250", _case(2, 24, 24, 4250, 4250, 64, dtype="fp16")),
        # A packed batch of prompts of 256 to 2 048 tokens.
        ("packed_32_prompts", _case(32, 32, 8, 2048, 2048, 128, causal=True, layout="NHD", entry="varlen", len_min=256, len_seed=5)),
        # The options together: fp16, one Q mean per head, a scale of the caller's own, the LSE wanted (ring composition).
        ("lse_8k", _case(2, 16, 16, 8192, 8192, 128, dtype="fp16", entry="lse", block_mean=False, scale=0.9)),
        # Language-model prefill at full batch: Llama-3-8B shape, 8 x 8 192 tokens.
        ("prefill_8x8k", _case(8, 32, 8, 8192, 8192, 128, causal=True, layout="NHD", k_dist="rope")),
        # A layer of the CogVideoX-5B-shaped video transformer: 226 text + 17 550 video tokens, 64-wide heads.
        ("video_17776", _case(2, 48, 48, 17776, 17776, 64, k_dist="outlier")),
        # The kernel benchmark the product is quoted on.
        ("bench_32k", _case(4, 32, 32, 32768, 32768, 128)),
        # A layer of the HunyuanVideo-shaped transformer, 720p x 129 frames: the longest sequence in use.
        ("video_119056", _case(1, 24, 24, 119056, 119056, 128)),
    ]
    return [dict(c, name=n) for n, c in named]


def draw(rng):
    """One more case of the same ranges."""
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def length(lo, hi):                   # every third one a multiple of 128
        n = span(lo, hi)
        return n if rng.random() < 2 / 3 else max(128, (n + 64) // 128 * 128)

    D = rng.choice((64, 128))
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    layout = rng.choice(("HND", "NHD"))
    kind = rng.choice(("self", "self", "self", "cross", "prefill", "prefill", "chunk", "decode", "packed"))
    if kind == "self":                    # image and video transformers
        n = length(1000, 60000)
        H = rng.choice((2, 8, 12, 16, 24, 32, 40, 48))
        B = rng.choice((1, 1, 2, 4))
        while 4 * B * H * n * n * D > 1.0e14 and B * H > 1:
            B, H = (B // 2, H) if B > 1 else (B, H // 2)
        lse = rng.random() < 0.25
        return _case(B, H, H, n, n, D, dtype, False, layout, rng.choice(("offset", "outlier")), "lse" if lse else "dense",
                     rng.random() < 0.75, rng.choice((1.0, 1.0, 0.9)))
    if kind == "cross":
        H = rng.choice((12, 24, 40, 48))
        return _case(rng.choice((1, 2)), H, H, length(1000, 30000), length(64, 600), D, dtype, False, layout)
    Hq, group = rng.choice(((16, 2), (28, 7), (32, 4), (32, 1), (40, 5), (64, 8)))
    Hkv = Hq // group
    if kind == "prefill":
        n = length(500, 16000)
        B = rng.choice((1, 1, 2, 4, 8))
        return _case(B, Hq, Hkv, n, n, D, dtype, True, layout, "rope")
    if kind == "chunk":
        nq = length(128, 2048)
        return _case(rng.choice((1, 1, 2)), Hq, Hkv, nq, nq + length(1000, 30000), D, dtype, True, layout, "rope")
    if kind == "decode":
        return _case(rng.choice((1, 2, 4, 8, 16)), Hq, Hkv, rng.choice((1, 1, 1, 4)), length(1000, 16000), D, dtype, True, layout, "rope")
    n = length(500, 4000)
    return _case(rng.randint(3, 32), Hq, Hkv, n, n, D, dtype, True, "NHD", "rope", "varlen", len_min=max(1, n // 8), len_seed=rng.randrange(1 << 20))


def _lengths(case):
    """The lengths of a packed batch, the same for every seed of the inputs."""
    r = random.Random(case["len_seed"])
    lens = [r.randint(case["len_min"], case["Nq"]) for _ in range(case["B"])]
    lens[r.randrange(case["B"])] = case["Nq"]
    return lens


def _rope(x, pos):
    """Rotates [..., tokens, heads, D] by position (halves convention)."""
    half = x.shape[-1] // 2
    freq = 500000.0 ** (-torch.arange(half, device=x.device, dtype=torch.float32) / half)
    ang = (pos.float()[:, None] * freq)[:, None, :]
    c, s = ang.cos(), ang.sin()
    a, b = x[..., :half].float(), x[..., half:].float()
    return torch.cat((a * c - b * s, b * c + a * s), dim=-1).to(x.dtype)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    dt = _DTYPES[case["dtype"]]
    B, Hq, Hkv, Nq, Nk, D = (case[n] for n in ("B", "Hq", "Hkv", "Nq", "Nk", "D"))
    packed = case["entry"] == "varlen"
    if packed:
        lens = _lengths(case)
        total = sum(lens)
        shapes = [(total, h, D) for h in (Hq, Hkv, Hkv)]
    elif case["layout"] == "HND":
        shapes = [(B, Hq, Nq, D), (B, Hkv, Nk, D), (B, Hkv, Nk, D)]
    else:
        shapes = [(B, Nq, Hq, D), (B, Nk, Hkv, D), (B, Nk, Hkv, D)]
    q, k, v = (torch.empty(s, dtype=dt, device=dev).normal_(generator=g) for s in shapes)
    if case["k_dist"] == "offset":
        off = torch.randn(Hkv, 1, D, device=dev, generator=g) * 2.5
        k += (off if not packed and case["layout"] == "HND" else off.transpose(0, 1)).to(dt)
    elif case["k_dist"] == "outlier":
        k[..., torch.randperm(D, device=dev, generator=g)[:4]] *= 2
    else:
        if packed:
            pos_q = pos_k = torch.cat([torch.arange(n, device=dev) for n in lens])
        else:
            pos_k = torch.arange(Nk, device=dev)
            pos_q = pos_k[Nk - Nq:]
        hnd = not packed and case["layout"] == "HND"
        q, k = ((_rope(x.transpose(1, 2), p).transpose(1, 2).contiguous() if hnd else _rope(x, p)) for x, p in ((q, pos_q), (k, pos_k)))
    state = dict(entry=case["entry"], q=q, k=k, v=v, kw=dict(is_causal=case["causal"]))
    if not case["block_mean"]:
        state["kw"]["per_block_mean"] = False
    if case["scale"] != 1.0:
        state["kw"]["sm_scale"] = case["scale"] * D ** -0.5
    if packed:
        cu = torch.tensor([0] + lens).cumsum(0).to(device=dev, dtype=torch.int32)
        state["cu"], state["longest"] = cu, max(lens)
    else:
        state["kw"]["tensor_layout"] = case["layout"]
    return state


def run(state):
    q, k, v, kw = state["q"], state["k"], state["v"], state["kw"]
    if state["entry"] == "varlen":
        return sageattn_varlen(q, k, v, state["cu"], state["cu"], state["longest"], state["longest"], **kw)
    if state["entry"] == "lse":
        return sageattn(q, k, v, return_lse=True, **kw)
    return sageattn3(q, k, v, **kw)


def work(case):
    """Each of q, k, v read once, the output (and LSE) written once; 4 D operations per visible (query, key) pair."""
    B, Hq, Hkv, Nq, Nk, D = (case[n] for n in ("B", "Hq", "Hkv", "Nq", "Nk", "D"))

    def pairs(nq, nk):
        if not case["causal"]:
            return nq * nk
        first = nk - nq + 1               # keys the first query row sees; one more in every row
        return nq * first + nq * (nq - 1) // 2 if first >= 0 else nk * (nk + 1) // 2

    lens = [(n, n) for n in _lengths(case)] if case["entry"] == "varlen" else [(Nq, Nk)] * B
    q_rows, k_rows = sum(a for a, _ in lens) * Hq, sum(b for _, b in lens) * Hkv
    return {"bytes": 2 * D * (2 * q_rows + 2 * k_rows) + (4 * q_rows if case["entry"] == "lse" else 0),
            "flops": 4 * D * Hq * sum(pairs(a, b) for a, b in lens)}


def tolerance(case):
    """Outputs are 16-bit, computed through four-bit operands: an exponential that is off in its last bit moves a code of
    P, or its eight-bit block scale, by a step where it lies on a rounding boundary."""
    return {"rel": 1e-2}
