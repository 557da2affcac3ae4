"""The attention work of a diffusion transformer as a program hands it to dtb200, for timing.

Sequences are laid out ``[image or video tokens | text tokens]`` with the padding at the end, heads are 128 wide, q and k
are RMS-normed per head, and everything a call returns is bf16.  The sizes are those of ``dtb200.inputs.CONFIGS`` and of
the shards that 8 GPUs hold of them, whole and ragged.  A case is one of:

  attention  ``dtb200.attention`` on q, k, v and the valid lengths
  bounded    ``dtb200.sdpa(use_fixed_m=True)``: keys smoothed, per-head bound taken, constant-offset softmax
  fp8        ``dtb200.attention(qk_fp8=True)``: q and k cast to E4M3 for the score product
  ring       key/value shards folded one after the other into a running state, which is then normalised
  block      the attention half of a DiT block: ``qk_prepass`` on the projections, ``attention``, ``out_proj``
  sparse     ``dtb200.sparse_attention`` with a window around each query block and all text keys

``pad`` padded positions trail the last batch element, and evenly fewer the ones before it.
"""
import math
import os
import sys

import torch

sys.path.insert(1, os.path.join(os.getcwd(), "diffusers-tpu_b200"))
import dtb200  # noqa: E402

D = 128
TEXT = 512          # text tokens at the end of a sequence


def listed():
    def case(name, op, B, H, S, Skv=0, pad=0, **more):
        return {"name": name, "op": op, "B": B, "H": H, "S": S, "Skv": Skv or S, "pad": pad, **more}

    return [
        # one layer call of a 512 x 512 image on one of 8 GPUs (3 of 24 heads): the smallest call, all latency
        case("image512_shard8", "attention", 1, 3, 1280, pad=37),
        # the same call on one GPU: one wave of blocks, host and launch time in view
        case("image512", "attention", 1, 24, 1280, pad=37),
        # a 1024 x 1024 image, both guidance branches: the everyday call
        case("image1024", "attention", 2, 24, 4608, pad=300),
        # the same call on one of 8 GPUs (guidance branches and heads split): fewer blocks than the chip has SMs
        case("image1024_shard8", "attention", 1, 6, 4608, pad=150),
        # a 2048 x 2048 image
        case("image2048", "attention", 2, 24, 16896, pad=211),
        # a 480p clip of 121 frames: the longest sequence that one GPU commonly gets whole
        case("video480p", "attention", 2, 40, 48872, pad=77),
        # a few queries against a long sequence (refreshed text or register tokens), ragged on both sides
        case("short_query", "attention", 2, 24, 333, Skv=16731, pad=211),
        # the 1024 x 1024 call with bounded logits, smoothing and bound included
        case("image1024_bounded", "bounded", 2, 24, 4608, pad=300),
        # the 2048 x 2048 call with 8-bit scores, casts included
        case("image2048_fp8", "fp8", 2, 24, 16896, pad=211),
        # two steps of the ring that spreads a 768p clip of 345 frames over 8 GPUs
        case("video768p_ring", "ring", 1, 40, 43912, pad=77, steps=2),
        # one DiT block's attention half on a 1024 x 1024 image: projections in, hidden states out
        case("image1024_block", "block", 2, 24, 4608, pad=300, rotary=96),
        # a 480p clip with a temporal window of six latent frames to either side
        case("video480p_sparse", "sparse", 1, 40, 48872, pad=77, window=9360),
    ]


def draw(rng):
    op = rng.choice(["attention", "attention", "attention", "short", "bounded", "fp8", "ring", "block", "sparse"])

    def log_uniform(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    B = rng.choice([1, 2])
    H = rng.choice([1, 2, 3, 5, 6, 10, 12, 20, 24, 40])
    S = log_uniform(1024, 48872)
    if rng.random() < 0.4:
        S -= S % 128                      # whole tiles as often as ragged ones
    case = {"op": op, "B": B, "H": H, "S": S, "Skv": S, "pad": rng.randint(0, 300)}
    if op == "short":
        case.update(op="attention", S=rng.randint(64, 768))
    elif op == "ring":
        case.update(S=min(S, 24436), steps=rng.choice([2, 3, 4]))
        case["Skv"] = case["S"]
    elif op == "block":
        case.update(S=min(S, 16896), H=max(H, 6), rotary=rng.choice([64, 96, 128]))
        case["Skv"] = case["S"]
    elif op == "sparse":
        case["window"] = log_uniform(256, S)
    return case


def _kv_len(case):
    """Valid length of each batch element of the whole sequence (all shards of a ring together)."""
    total = case["Skv"] * case.get("steps", 1)
    return [total - case["pad"] * (b + 1) // case["B"] for b in range(case["B"])]


def _table(case):
    """Key blocks of 128 that each block of 256 queries visits: its window, and the text at the end."""
    n_q, n_kv = -(-case["S"] // 256), -(-case["S"] // 128)
    text = range(max(case["S"] - TEXT, 0) // 128, n_kv)
    rows = []
    for qb in range(n_q):
        lo = max(256 * qb - case["window"], 0) // 128
        hi = min((256 * qb + 255 + case["window"]) // 128, n_kv - 1)
        rows.append(sorted(set(range(lo, hi + 1)) | set(text)))
    return rows


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, H, S, Skv = case["B"], case["H"], case["S"], case["Skv"]

    def normal(*shape):
        return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)

    def normed(*shape):
        x = normal(*shape)
        return x.mul_(torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6)).to(torch.bfloat16)

    state = {"case": case, "kv_len": torch.tensor(_kv_len(case), dtype=torch.int32, device="cuda")}
    if case["op"] == "block":
        # the q, k, v projections lie in one [B, S, 3 * H * 128] tensor, as a fused linear layer leaves them
        qkv = normal(B, S, 3 * H * D).to(torch.bfloat16)
        state["q"], state["k"], state["v"] = (t.unflatten(-1, (H, D)) for t in qkv.chunk(3, dim=-1))
        state["weights"] = [1.0 + 0.1 * normal(D) for _ in range(2)]
        half = case["rotary"] // 2
        inv = 10000.0 ** (-torch.arange(half, device="cuda", dtype=torch.float32) / half)
        angle = torch.arange(S, device="cuda", dtype=torch.float32)[:, None] * inv[None, :]
        state["rope"] = (torch.cat([angle.cos()] * 2, -1), torch.cat([angle.sin()] * 2, -1))
        state["w_out"] = (normal(H * D, H * D) * (H * D) ** -0.5).to(torch.bfloat16)
        return state
    state["q"] = normed(B, H, S, D)
    if case["op"] == "ring":
        state["shards"] = [(normed(B, H, Skv, D), normal(B, H, Skv, D).to(torch.bfloat16)) for _ in range(case["steps"])]
        state["running"] = dtb200.ResidualState(B, H, S, state["q"].device)
        return state
    state["k"] = normed(B, H, Skv, D)
    state["v"] = normal(B, H, Skv, D).to(torch.bfloat16)
    if case["op"] == "sparse":
        state["table"] = dtb200.make_block_table(_table(case), seq_q=S, seq_kv=Skv, block_q=256, block_kv=128)
    return state


def run(state):
    case, op, kv_len, q = state["case"], state["case"]["op"], state["kv_len"], state["q"]
    if op == "attention":
        # queries of the sequence itself are padded where its keys are; queries from elsewhere are all live
        return dtb200.attention(q, state["k"], state["v"], kv_len=kv_len, zero_padded_rows=case["S"] == case["Skv"])
    if op == "bounded":
        return dtb200.sdpa(q, state["k"], state["v"], kv_len=kv_len, use_fixed_m=True)
    if op == "fp8":
        return dtb200.attention(q, state["k"], state["v"], kv_len=kv_len, qk_fp8=True)
    if op == "ring":
        running = state["running"]
        running.fresh = True
        for i, (k, v) in enumerate(state["shards"]):
            dtb200.residual_attention_(running, q, k, v, kv_len=kv_len, kv_offset=i * case["Skv"])
        return dtb200.finalize_residual(running, kv_len=kv_len)
    if op == "block":
        wq, wk = state["weights"]
        qn, kn, vn, _ = dtb200.qk_prepass(q, state["k"], state["v"], q_weight=wq, k_weight=wk, rope=state["rope"], kv_len=kv_len)
        return dtb200.out_proj(dtb200.attention(qn, kn, vn, kv_len=kv_len), state["w_out"])
    return dtb200.sparse_attention(q, state["k"], state["v"], kv_table=state["table"], kv_len=kv_len)


def work(case):
    """Each tensor of the call moved once; multiplications for the valid queries and keys only."""
    B, H, S, op = case["B"], case["H"], case["S"], case["op"]
    lens = _kv_len(case)
    self_attention = S == case["Skv"]
    rows = [min(n, S) if self_attention else S for n in lens]
    pairs = sum(r * n for r, n in zip(rows, lens))
    if op == "sparse":
        pairs = sum(max(min(256, rows[b] - 256 * qb), 0) * sum(max(min(128, lens[b] - 128 * t), 0) for t in tiles)
                    for b in range(B) for qb, tiles in enumerate(_table(case)))
    flops = 4.0 * H * D * pairs
    moved = 2.0 * H * D * (B * S + sum(rows) + 2 * sum(lens))     # o whole; q, k and v where they are valid
    if op == "block":
        hidden = H * D
        flops += 2.0 * B * S * hidden * hidden
        moved += 2.0 * hidden * hidden + 8.0 * S * case["rotary"]
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """bf16 results over bf16 probabilities, rounding alone.  Against float32 throughout, calls show rel 2.3e-3 to 2.8e-3 and
    max 9e-3 to 1.8e-2; two correct implementations may be both that far off."""
    return {"rel": 1e-2, "max": 0.1}


# Beyond this many (query, key) pairs over all heads the 64-bit scores take too long.
_EXACT_PAIRS = 5e10


def exact(case, seed):
    """What ``run`` returns, in 64 bits from the same inputs: one head and a slice of the queries at a time."""
    B, H, S, op = case["B"], case["H"], case["S"], case["op"]
    total = case["Skv"] * case.get("steps", 1)
    if float(B) * H * S * total > _EXACT_PAIRS:
        return None
    state = prepare(case, seed)
    lens, f64 = _kv_len(case), torch.float64
    q, scale = state["q"], D ** -0.5
    if op == "ring":
        k, v = (torch.cat(shards, dim=2) for shards in zip(*state["shards"]))
    else:
        k, v = state["k"], state["v"]
    if op == "block":
        cos, sin = (t.to(f64) for t in state["rope"])
        half = case["rotary"] // 2

        def finished(x, weight):
            x = x.transpose(1, 2).to(f64)
            x = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * weight.to(f64)
            head, rest = x[..., :2 * half], x[..., 2 * half:]
            turned = torch.cat([-head[..., half:], head[..., :half]], -1)
            return torch.cat([head * cos + turned * sin, rest], -1)

        q, k, v = finished(q, state["weights"][0]), finished(k, state["weights"][1]), v.transpose(1, 2)
    elif op == "fp8":
        def cast(x, by):
            return (x.float() * by).clamp(-448, 448).to(torch.float8_e4m3fn)

        q, k, scale = cast(q, scale / math.log(2)), cast(k, 1.0), math.log(2)
    out = torch.zeros(B, H, S, D, dtype=f64, device="cuda")
    table = _table(case) if op == "sparse" else None
    rows = 256 if table else max(256, min(4096, int(3e8) // total))
    for b in range(B):
        last = min(lens[b], S) if S == case["Skv"] or op == "ring" else S
        for h in range(H):
            k64, v64 = k[b, h, :lens[b]].to(f64), v[b, h, :lens[b]].to(f64)
            for lo in range(0, last, rows):
                hi = min(lo + rows, last)
                kk, vv = k64, v64
                if table:
                    tiles = torch.tensor(table[lo // 256], device="cuda")
                    keys = (tiles[:, None] * 128 + torch.arange(128, device="cuda")).flatten()
                    keys = keys[keys < lens[b]]
                    kk, vv = k64[keys], v64[keys]
                p = torch.softmax((q[b, h, lo:hi].to(f64) @ kk.T).mul_(scale), -1)
                out[b, h, lo:hi] = p @ vv
    if op == "block":
        return out.transpose(1, 2).reshape(B, S, H * D) @ state["w_out"].to(f64)
    return out
