"""What a user of this package has it do: the self-attention calls of a causal video DiT.

Five kinds of call, each through the package's public entry points:

  layer    self_attention_kv: one layer call of the KV-cache rollout, from the raw projections (RMSNorm, RoPE, cache
           write, attention, cache bookkeeping).  Every layer of every denoising step makes one.
  dropin   monarch_attn_with_kv_cache: the same attention with the reference's call signature (q, k rotated already).
  train    monarch_attn_with_kv_cache under autograd: forward, then the gradients of the queries and of the new keys
           and values (grad_only_new_kv, as the self-forcing training rollout calls it).
  clip     monarch_attn: no cache, block-causal over chunks (or unmasked), a whole clip at once.
  dense    self_attention_kv with dense attention (the "regular" configuration and the dense first chunk).

Fields of a case: B videos, H heads (of 128), a token grid of h x w per latent frame, `frames` new frames per call,
`cached` frames visible to the call (the new ones included), the blocking (f_tied, h_reduce, w_reduce) and
num_iters.  `window` > 0: a sliding window of that many frames with `sink` frames kept; every call then brings a new
chunk into a full window, so the oldest frames are evicted.  All tensors are bf16, N(0, 1) as the normalised
projections are.
"""
import torch

import self_forcing_b200 as sfb

D = 128


def _case(name, kind, B, H, h, w, frames, cached, blocking=(1, 1, 1), iters=1, window=0, sink=0, causal=False):
    c = {"kind": kind, "B": B, "H": H, "h": h, "w": w, "frames": frames, "cached": cached, "f_tied": blocking[0],
         "h_reduce": blocking[1], "w_reduce": blocking[2], "iters": iters, "window": window, "sink": sink,
         "causal": causal}
    return dict(c, name=name) if name else c


def listed():
    tied3, reduce2xh, reduce4xw2xh = (3, 1, 1), (1, 2, 1), (1, 2, 4)
    return [
        # A one-frame chunk of a thumbnail grid, two heads: as small as a call gets; launches and host time are all of it.
        _case("layer_thumbnail", "layer", 1, 2, 6, 8, 1, 4),
        # First chunk of a 480p rollout (30 x 52 tokens a frame, 12 heads): the cache holds nothing else yet.
        _case("layer_first_chunk", "layer", 1, 12, 30, 52, 3, 3),
        # Middle of the rollout with three frames tied into one Monarch group.
        _case("layer_tied3frame", "layer", 1, 12, 30, 52, 3, 12, tied3),
        # Last chunk of the rollout: 4680 queries against 32760 cached tokens.
        _case("layer_last_chunk", "layer", 1, 12, 30, 52, 3, 21),
        # The same layer call of the large model, all 40 heads on one GPU.
        _case("layer_40_heads", "layer", 1, 40, 30, 52, 3, 21),
        # Long video: a full 12-frame window that keeps 3 sink frames and evicts 3 frames for each new chunk.
        _case("layer_sliding_window", "layer", 1, 12, 30, 52, 3, 12, window=12, sink=3),
        # Dense attention in the middle of the rollout (the configuration that Monarch is compared with).
        _case("dense_mid_rollout", "dense", 1, 12, 30, 52, 3, 12),
        # Several videos at once behind the reference's call signature, frames split into two bands of rows.
        _case("dropin_batch_reduce2xh", "dropin", 4, 12, 30, 52, 3, 9, reduce2xh),
        # The finest blocking that the configurations use, at the end of the rollout.
        _case("dropin_reduce4xw2xh", "dropin", 1, 12, 30, 52, 3, 21, reduce4xw2xh),
        # The iterative ("slow") variant with its 20 alternating passes, first chunk.
        _case("dropin_20_passes", "dropin", 1, 12, 30, 52, 3, 3, iters=20),
        # A training step's attention call: forward and backward, gradients of q and of the new keys / values.
        _case("train_mid_rollout", "train", 1, 12, 30, 52, 3, 12),
        # A whole 12-frame clip without a cache, causal over 3-frame chunks.
        _case("clip_block_causal", "clip", 1, 12, 30, 52, 12, 12, causal=True),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    """Another case of the same ranges: grids from 6 x 8 tokens to 45 x 80 (720p), 1 to 40 heads, 1 to 21 cached
    frames, every blocking; no larger than the largest listed case of its kind (by `_size`)."""
    while True:
        kind = rng.choice(["layer", "layer", "layer", "dropin", "dropin", "iter", "train", "clip", "dense"])
        if rng.random() < 0.4:
            h, w = 30, 52
        else:
            h, w = _log(rng, 6, 45), _log(rng, 8, 80)
        H = rng.choice([1, 2, 3, 5, 10, 12, 12, 16, 40])
        B = rng.choice([1, 1, 1, 2, 3, 4])
        f_tied = rng.choice([1, 1, 1, 3])
        h_reduce = rng.choice([d for d in (1, 1, 2, 3) if h % d == 0])
        w_reduce = rng.choice([d for d in (1, 1, 2, 4) if w % d == 0])
        if f_tied == 3 and kind == "train":
            h_reduce = 1
        frames = rng.choice([3, 3, 3, 1, 2]) if f_tied == 1 else 3
        cached = frames * rng.randint(1, 21 // frames)
        window = sink = 0
        if kind == "layer" and frames == 3 and cached >= 6 and rng.random() < 0.3:
            window, sink = cached, 3 * rng.randint(0, cached // 3 - 2)
        iters = rng.randint(2, 20) if kind == "iter" else 1
        causal = kind == "clip" and cached % 3 == 0 and rng.random() < 0.7
        if kind == "clip":
            frames = cached
        b1, b2 = f_tied * h // h_reduce, w // w_reduce
        if b1 > 96 or b2 < 4 or (b2 > 64 and kind in ("iter", "train")):
            continue
        c = _case(None, "dropin" if kind == "iter" else kind, B, H, h, w, frames, cached, (f_tied, h_reduce, w_reduce),
                  iters, window, sink, causal)
        if _size(c) <= max(_size(x) for x in listed() if _same_kind(c, x)):
            return c


def _same_kind(c, x):
    return c["kind"] == x["kind"] and (c["iters"] > 1) == (x["iters"] > 1)


def _block(c):
    """(b1, b2): rows and columns of a Monarch block."""
    return c["f_tied"] * c["h"] // c["h_reduce"], c["w"] // c["w_reduce"]


def _tokens(c):
    """(queries, keys) of a call, per video and head."""
    frame = c["h"] * c["w"]
    return c["frames"] * frame, c["cached"] * frame


def _size(c):
    """How large a case is beside others of its kind: the row results of the Monarch step, weighted with the lengths of
    the dot products' other side, or the dense logits."""
    n_q, n_kv = _tokens(c)
    pairs = c["B"] * c["H"] * n_q * n_kv
    if c["kind"] == "dense":
        return pairs
    b1, b2 = _block(c)
    return c["iters"] * pairs / (b1 * b2) * (128 + b1 + b2)


def _blocking(c):
    return c["f_tied"], c["h_reduce"], c["w_reduce"], c["h"], c["w"]


def prepare(case, seed):
    c = dict(case)
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device=dev, dtype=torch.bfloat16)

    B, H, h, w = c["B"], c["H"], c["h"], c["w"]
    n_q, n_kv = _tokens(c)
    s = {"case": c, "q": randn(B, n_q, H, D), "k": randn(B, n_q, H, D), "v": randn(B, n_q, H, D)}
    if c["kind"] == "clip":
        return s
    # The cache is one buffer per layer for the whole rollout; a call sees the part written so far.
    n_buf = n_kv if c["window"] else max(n_kv, 21 * h * w)
    k_buf, v_buf = randn(B, n_buf, H, D), randn(B, n_buf, H, D)
    if c["kind"] in ("layer", "dense"):
        past = n_kv if c["window"] else n_kv - n_q
        s["cache"] = sfb.KVCache(k_buf, v_buf, past, past)
        s["past"] = past
        s["cfg"] = sfb.LayerConfig(use_framewise=c["f_tied"] == 1, h_reduce=c["h_reduce"], w_reduce=c["w_reduce"],
                                   num_iters=c["iters"], disable_monarch=c["kind"] == "dense",
                                   local_attn_size=c["window"] or -1, sink_size=c["sink"], max_attention_size=n_buf)
        s["norm_q"], s["norm_k"] = 1 + 0.1 * randn(H * D), 1 + 0.1 * randn(H * D)
    else:
        s["k_buf"], s["v_buf"] = k_buf, v_buf
    if c["kind"] == "train":
        for name in ("q", "k", "v"):
            s[name].requires_grad_()
        s["d_out"] = randn(B, n_q, H, D)
    return s


def run(s):
    c = s["case"]
    n_q, n_kv = _tokens(c)
    if c["kind"] in ("layer", "dense"):
        cache = s["cache"]
        if c["window"]:
            cache.global_end = cache.local_end = s["past"]      # the next chunk of a window that is full
        with torch.no_grad():
            out = sfb.self_attention_kv(s["q"], s["k"], s["v"], cache, s["past"], (c["frames"], c["h"], c["w"]),
                                        s["cfg"], norm_q_weight=s["norm_q"], norm_k_weight=s["norm_k"])
        return {"out": out, "k_cache": cache.k, "v_cache": cache.v}
    if c["kind"] == "clip":
        with torch.no_grad():
            return sfb.monarch_attn(s["q"], s["k"], s["v"], *_blocking(c), num_iters=c["iters"],
                                    block_causal_size=3 * c["h"] * c["w"] if c["causal"] else None)
    args = (s["q"], s["k_buf"][:, :n_kv], s["v_buf"][:, :n_kv], s["k"], s["v"], n_kv - n_q, n_kv, *_blocking(c))
    if c["kind"] == "dropin":
        with torch.no_grad():
            out = sfb.monarch_attn_with_kv_cache(*args, num_iters=c["iters"])
        return {"out": out, "k_cache": s["k_buf"], "v_cache": s["v_buf"]}
    out = sfb.monarch_attn_with_kv_cache(*args, grad_only_new_kv=True)
    grads = torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["d_out"])
    return {"out": out, "grads": grads, "k_cache": s["k_buf"], "v_cache": s["v_buf"]}


def work(case):
    """Matrix products of the two Monarch steps (3 / b1 and 2 / b2 of a dense product's n_q x n_kv x D each), every
    input read once and every output written once.  A pass of the iterative variant before the last has 2 / b1 and
    2 / b2.  The backward repeats no forward product here: twice the forward's, less what grad_only_new_kv leaves out."""
    c = case
    B, H = c["B"], c["H"]
    n_q, n_kv = _tokens(c)
    b1, b2 = _block(c)
    row = 2 * H * D * B                                         # bytes of one token of one tensor, all videos
    product = 2.0 * B * H * D * n_q * n_kv
    if c["kind"] == "clip":
        if c["causal"]:
            chunks = -(-c["frames"] // 3)
            product *= (chunks + 1) / (2 * chunks)
        return {"bytes": 4 * n_q * row, "flops": product * (3 / b1 + 2 / b2)}
    # q, k, v in; the cached tokens read; the new slot and the output written
    nbytes = (3 * n_q + (n_kv - n_q) * 2 + 2 * n_q + n_q) * row
    if c["window"]:
        moved = n_kv - n_q - c["sink"] * c["h"] * c["w"]
        nbytes += 2 * max(0, moved) * row
    if c["kind"] == "dense":
        return {"bytes": nbytes, "flops": 2 * product}
    flops = product * (3 / b1 + 2 / b2) + (c["iters"] - 1) * product * (2 / b1 + 2 / b2)
    if c["kind"] == "train":
        nbytes += 4 * n_q * row                                 # d_out in, three gradients out
        flops += product * (3 / b1 + 4 / b2) + product * n_q / n_kv * 3 / b1
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # bf16 inputs and results, bf16 row results between the two steps; the gradients pass through two more such steps
    return {"rel": 2e-2 if case["kind"] == "train" else 1e-2, "max": 0.2}
