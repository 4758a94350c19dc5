"""What this framework is timed on: its attention, recurrence and expert calls as a serving step makes them, and a whole decode step of
its engine, each over the range of sizes that it is used at.

A case names its ``kind``; the functions of a kind are collected in ``KINDS`` at the end of the file.  Lengths of sequences follow from
the case alone (``mix`` seeds them), values and the order of cache blocks from the seed of ``prepare``.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from llm_from_scratch_b200 import ops
from llm_from_scratch_b200.workloads import c5_prefill_lengths, deal_blocks

DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}


# ------------------------------------------------------------------------------------------------ shared pieces
def _lengths(case: dict) -> np.ndarray:
    """Tokens of every sequence: ``spread`` names the distribution over [lo, hi]."""
    n, lo, hi = case["seqs"], case["lo"], case["hi"]
    rng = np.random.default_rng(case["mix"])
    if case["spread"] == "uniform":
        return rng.integers(lo, hi + 1, size=n).astype(np.int64)
    if case["spread"] == "log":
        return np.clip(np.rint(np.exp(rng.uniform(math.log(lo), math.log(hi), size=n))), lo, hi).astype(np.int64)
    return c5_prefill_lengths(num_seqs=n, total=case["total"], lo=lo, hi=hi, seed=case["mix"])


class _Draw:
    """Seeded normal and uniform tensors on the GPU."""

    def __init__(self, seed: int):
        self.device = torch.device("cuda")
        self.gen = torch.Generator(device=self.device).manual_seed(seed)
        self.order = np.random.default_rng(seed)          # of cache blocks and state slots

    def normal(self, *shape, dtype=torch.bfloat16, mean=0.0, std=1.0):
        out = torch.empty(shape, dtype=dtype, device=self.device)
        flat = out.view(-1)
        for at in range(0, flat.numel(), 1 << 28):        # a pool at a time would need its fp32 copy at once
            part = flat[at:at + (1 << 28)]
            part.copy_(torch.randn(part.numel(), generator=self.gen, device=self.device).mul_(std).add_(mean))
        return out

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=torch.float32):
        return (lo + (hi - lo) * torch.rand(*shape, generator=self.gen, device=self.device)).to(dtype)

    def ints(self, values, dtype):
        return torch.as_tensor(np.asarray(values), dtype=dtype).to(self.device)

    def blocks(self, lens, page: int):
        """Block tables over a shuffled pool, every sequence's slots in order, and the number of blocks."""
        dealt = deal_blocks(lens, page, self.order, pad_blocks=4)
        slots = np.concatenate([dealt.block_tables[i, np.arange(n) // page].astype(np.int64) * page + np.arange(n) % page
                                for i, n in enumerate(lens)])
        return self.ints(dealt.block_tables, torch.int32), self.ints(slots, torch.int64), dealt.num_blocks

    def offsets(self, lens):
        return self.ints(np.concatenate([[0], np.cumsum(lens)]), torch.int32)


def _attend(q, k, v, scale: float, first: int, rows: int = 0):
    """Causal attention in 64 bits: q [nq, H, d] at positions first .., k [nk, G, d], v [nk, G, dv]."""
    nq, H, d = q.shape
    G = k.shape[1]
    k, v = k.double().permute(1, 2, 0), v.double().transpose(0, 1)                       # [G, d, nk], [G, nk, dv]
    out = torch.empty(nq, H, v.shape[-1], dtype=torch.float64, device=q.device)
    rows = rows or max(1, (1 << 27) // (H * max(1, k.shape[2])))
    for at in range(0, nq, rows):
        part = q[at:at + rows].double()
        n, seen = part.shape[0], min(k.shape[2], first + at + part.shape[0])
        part = part.view(n, G, H // G, d).permute(1, 2, 0, 3).reshape(G, -1, d)
        s = (part @ k[..., :seen]).mul_(scale).view(G, H // G, n, seen)
        i = torch.arange(first + at, first + at + n, device=q.device)[:, None]
        s.masked_fill_(torch.arange(seen, device=q.device)[None] > i, -math.inf)
        s = torch.softmax(s, -1).view(G, -1, seen)
        out[at:at + n] = (s @ v[:, :seen]).view(G, H // G, n, -1).permute(2, 0, 1, 3).reshape(n, H, -1)
    return out


def _cached(pool, table, n: int):
    """The first n rows of a sequence in a paged pool."""
    page = pool.shape[1]
    return pool[table[:(n + page - 1) // page].long()].flatten(0, 1)[:n]


# ------------------------------------------------------------------------------------------------ decode attention
# One new token per sequence over a paged cache: what every decode step runs in every layer.  From a single request to full
# batches, contexts from a short chat to 8192 tokens; bf16, and fp32 for the engine's fp32 mode.
def _prepare_decode(case, seed):
    d, dt, lens = _Draw(seed), DTYPES[case["dtype"]], _lengths(case)
    tables, _, blocks = d.blocks(lens, case["page"])
    pool = (blocks, case["page"], case["kv_heads"], case["dim"])
    return dict(q=d.normal(len(lens), case["heads"], case["dim"], dtype=dt), k=d.normal(*pool, dtype=dt), v=d.normal(*pool, dtype=dt),
                tables=tables, lens=d.ints(lens, torch.int64), scale=case["dim"] ** -0.5)


def _run_decode(s):
    return ops.paged_decode_gqa(s["q"], s["k"], s["v"], s["tables"], s["lens"], s["scale"])


def _exact_decode(case, seed):
    s = _prepare_decode(case, seed)
    return torch.cat([_attend(s["q"][i:i + 1], _cached(s["k"], s["tables"][i], n), _cached(s["v"], s["tables"][i], n), s["scale"], n - 1)
                      for i, n in enumerate(map(int, _lengths(case)))])


def _work_decode(case):
    lens, size = _lengths(case), 4 if case["dtype"] == "f32" else 2
    read = int(lens.sum()) * 2 * case["kv_heads"] * case["dim"] * size + int((-(-lens // case["page"])).sum()) * 4
    return {"bytes": read + len(lens) * (2 * case["heads"] * case["dim"] * size + 8),
            "flops": int(lens.sum()) * 4 * case["heads"] * case["dim"]}


def _draw_decode(rng):
    if rng.random() < 0.6:
        heads, kv, dim = rng.choice([(16, 4, 64), (32, 8, 128)])
        dtype, page, seqs, hi = "bf16", rng.choice([16, 64, 256]), _log(rng, 1, 256), _log(rng, 64, 8192)
    else:
        heads, kv, dim = rng.choice([(16, 4, 32), (16, 4, 64), (32, 8, 128)])
        dtype, page, seqs, hi = "f32", 16, _log(rng, 1, 128), _log(rng, 32, 2048)
    return dict(kind="decode", dtype=dtype, heads=heads, kv_heads=kv, dim=dim, page=page, seqs=seqs, spread=rng.choice(["uniform", "log"]),
                lo=max(1, hi // rng.choice([1, 8, 64])), hi=hi, mix=rng.randrange(1 << 20))


# ------------------------------------------------------------------------------------------------ prompt attention
# Causal attention over packed prompts, with the new keys and values written into the paged cache in the same call: what a
# prefill step runs in every layer.  The tile list is made once per step and shared by the layers.
def _prepare_prompts(case, seed):
    d, dt, lens = _Draw(seed), DTYPES[case["dtype"]], _lengths(case)
    H, G, D, T = case["heads"], case["kv_heads"], case["dim"], int(lens.sum())
    _, slots, blocks = d.blocks(lens, 16)
    cu, longest = d.offsets(lens), int(lens.max())
    q, k, v = d.normal(T, H, D, dtype=dt), d.normal(T, G, D, dtype=dt), d.normal(T, G, D, dtype=dt)
    caches = [torch.zeros(blocks, 16, G, D, dtype=dt, device="cuda") for _ in range(2)]
    plan = ops.prefill_plan(cu, T, longest, ops.prefill_tile_rows(H, G, D, D, dt))
    return dict(q=q, k=k, v=v, cu=cu, longest=longest, scale=D ** -0.5, caches=caches, slots=slots, plan=plan)


def _run_prompts(s):
    k_cache, v_cache = s["caches"]
    o = ops.prefill_varlen(s["q"], s["k"], s["v"], s["cu"], s["cu"], s["longest"], s["longest"], s["scale"], k_cache, v_cache,
                           plan=s["plan"], slot_mapping=s["slots"])
    return [o, k_cache, v_cache]


def _exact_prompts(case, seed):
    s, lens = _prepare_prompts(case, seed), _lengths(case)
    out = torch.empty(s["q"].shape, dtype=torch.float64, device="cuda")
    at = 0
    for n in map(int, lens):
        out[at:at + n] = _attend(*(s[x][at:at + n] for x in "qkv"), s["scale"], 0)
        at += n
    return [out, None, None]


def _work_prompts(case):
    lens, size = _lengths(case), 4 if case["dtype"] == "f32" else 2
    H, G, D, T = case["heads"], case["kv_heads"], case["dim"], int(lens.sum())
    return {"bytes": T * ((2 * H + 4 * G) * D * size + 8), "flops": int((lens * (lens + 1) // 2).sum()) * 4 * H * D}


def _draw_prompts(rng):
    if rng.random() < 0.6:
        heads, kv, dim = rng.choice([(16, 4, 64), (32, 8, 128)])
        dtype, total, hi = "bf16", _log(rng, 64, 65536), _log(rng, 32, 8192)
    else:
        heads, kv, dim = rng.choice([(16, 4, 32), (16, 4, 64), (32, 8, 128)])
        dtype, total, hi = "f32", _log(rng, 64, 8192), _log(rng, 16, 1024)
    lo = max(1, hi // rng.choice([1, 4, 16]))
    return dict(kind="prompts", dtype=dtype, heads=heads, kv_heads=kv, dim=dim, seqs=max(1, min(256, 2 * total // (lo + hi))), spread="uniform",
                lo=lo, hi=hi, mix=rng.randrange(1 << 20))


# ------------------------------------------------------------------------------------------------ latent decode attention
# The absorbed form of latent attention (rank 512, 64 rotary channels) over a paged pool of latent rows.
RANK, ROPE = 512, 64


def _prepare_latent(case, seed):
    d, lens, H = _Draw(seed), _lengths(case), case["heads"]
    tables, _, blocks = d.blocks(lens, case["page"])
    return dict(qa=d.normal(len(lens), H, RANK, std=0.3), qr=d.normal(len(lens), H, ROPE), rows=d.normal(blocks, case["page"], RANK + ROPE),
                tables=tables, lens=d.ints(lens, torch.int64), scale=192 ** -0.5)


def _run_latent(s):
    return ops.mla_decode(s["qa"], s["qr"], s["rows"], s["tables"], s["lens"], s["scale"])


def _exact_latent(case, seed):
    s = _prepare_latent(case, seed)
    q = torch.cat([s["qa"], s["qr"]], -1)
    rows = lambda i, n: _cached(s["rows"], s["tables"][i], n).unsqueeze(1)
    return torch.cat([_attend(q[i:i + 1], r, r[..., :RANK], s["scale"], n - 1)
                      for i, n in enumerate(map(int, _lengths(case))) for r in (rows(i, n),)])


def _work_latent(case):
    lens, H = _lengths(case), case["heads"]
    return {"bytes": int(lens.sum()) * (RANK + ROPE) * 2 + int((-(-lens // case["page"])).sum()) * 4
            + len(lens) * (H * (2 * RANK + ROPE) * 2 + 8), "flops": int(lens.sum()) * 2 * H * (2 * RANK + ROPE)}


def _draw_latent(rng):
    hi = _log(rng, 128, 16384)
    return dict(kind="latent_decode", heads=rng.choice([8, 16, 32]), page=rng.choice([16, 64]), seqs=_log(rng, 1, 256),
                spread=rng.choice(["uniform", "log"]), lo=max(1, hi // rng.choice([1, 8, 32])), hi=hi, mix=rng.randrange(1 << 20))


# ------------------------------------------------------------------------------------------------ the Nabalix mixer
# Talking-heads attention in a sliding window beside the gated recurrence, between the projection of the layer's input and the
# output projections; prompts (all tokens of whole prompts) or a decode step (one token per sequence behind a full window).
MIXERS = {1024: dict(H=16, G=4, D=64, rec=8, R=64, window=1024), 2048: dict(H=16, G=4, D=128, rec=16, R=128, window=1024),
          4096: dict(H=32, G=8, D=128, rec=16, R=128, window=2048)}


def _prepare_mixer(case, seed):
    d, lens, z = _Draw(seed), _lengths(case), MIXERS[case["width"]]
    H, G, D, rec, R, page = z["H"], z["G"], z["D"], z["rec"], z["R"], 64
    tables, slots, blocks = d.blocks(lens, page)
    n, decode = len(lens), case["stage"] == "decode"
    rows = n if decode else int(lens.sum())
    pool = (blocks, page, G, D)
    heads = ops.TalkingHeads(D ** -0.5, 30.0, d.uniform(H), d.uniform(H),
                             (torch.eye(H, device="cuda") + d.normal(H, H, dtype=torch.float32, std=0.2)).bfloat16(), z["window"], d.device)
    widths = dict(q=H * D, k=G * D, v=G * D, g=H * D, rq=rec * R, rf=rec * R, rv=rec * R)
    parts = dict(zip(widths, d.normal(rows, sum(widths.values())).split(list(widths.values()), 1)))
    s = dict(parts, heads=heads, tables=tables, eps=1e-5, bias=d.normal(rec * R, dtype=torch.float32, mean=3.0, std=1.5),
             lower=0.9 * d.uniform(rec * R), norm=d.normal(R, dtype=torch.float32, mean=1.0, std=0.1),
             state=d.normal(n + 2, rec, R, R, dtype=torch.float32), state_slots=d.ints(d.order.permutation(n + 2)[:n], torch.int64))
    if decode:
        last = np.cumsum(lens) - 1
        s.update(k_cache=d.normal(*pool), v_cache=d.normal(*pool), slots=slots[d.ints(last, torch.int64)].contiguous(),
                 where=dict(context_lens=d.ints(lens, torch.int64)), plan=None)
    else:
        cu = d.offsets(lens)
        s.update(k_cache=torch.zeros(pool, dtype=torch.bfloat16, device="cuda"), v_cache=torch.zeros(pool, dtype=torch.bfloat16, device="cuda"),
                 slots=slots, where=dict(cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=int(lens.max())),
                 plan=ops.prefill_plan(cu, rows, int(lens.max()), ops.TALKING_TILE_ROWS))
    return s


def _run_mixer(s):
    ops.store_kv_rows(s["k"], s["v"], s["k_cache"], s["v_cache"], s["slots"])
    left = ops.talking_attention(s["q"], s["g"], s["k_cache"], s["v_cache"], s["tables"], s["heads"], plan=s["plan"], **s["where"])
    right = ops.gated_recurrence(s["rq"], s["rf"], s["rv"], s["bias"], s["lower"], s["norm"], s["eps"], s["state"], s["state_slots"],
                                 **s["where"])
    return [left, right, s["state"], s["k_cache"], s["v_cache"]]


def _exact_mixer(case, seed):
    s, z, lens = _prepare_mixer(case, seed), MIXERS[case["width"]], _lengths(case)
    H, G, D, rec, R, decode = z["H"], z["G"], z["D"], z["rec"], z["R"], case["stage"] == "decode"
    c, rows, n = s["heads"], s["q"].shape[0], len(lens)
    q, gate = s["q"].double().view(rows, H, D), torch.sigmoid(s["g"].double()).view(rows, H, D)
    k, v = (s[x].double().view(rows, G, D) for x in "kv")
    talk, r1, r2 = (t.double() for t in (c.talk, c.r1, c.r2))
    left, at = torch.empty_like(q), 0
    for i, length in enumerate(map(int, lens)):
        if decode:
            keys, vals = (_cached(s[x + "_cache"], s["tables"][i], length).double() for x in "kv")
            keys[-1], vals[-1] = k[i], v[i]
            new = slice(i, i + 1)
        else:
            new = slice(at, at + length)
            keys, vals = k[new], v[new]
            at += length
        qs, first = q[new], length - (new.stop - new.start)
        for lo in range(0, qs.shape[0], 256):
            part = qs[lo:lo + 256]
            dist = torch.arange(first + lo, first + lo + part.shape[0], device="cuda")[:, None] - torch.arange(length, device="cuda")[None]
            m = torch.einsum("ighd,jgd->ghij", part.view(-1, G, H // G, D), keys).flatten(0, 1) * c.scale
            m = c.softcap * torch.tanh(m / c.softcap) - r1[:, None, None] * torch.log1p(r2[:, None, None] * dist.clamp(min=0))
            m = torch.einsum("hg,gij->hij", talk, m).masked_fill(((dist < 0) | (dist >= c.window))[None], -math.inf)
            p = torch.softmax(m, -1).view(G, H // G, -1, length)
            left[new][lo:lo + 256] = torch.einsum("ghij,jgd->ighd", p, vals).flatten(1, 2)
    left *= gate
    # the recurrence, token by token for all sequences at once
    rq = torch.nn.functional.silu(s["rq"].double()).view(rows, rec, R)
    low = s["lower"].double()
    f = (low + (1 - low) * torch.sigmoid(s["rf"].double() + s["bias"].double())).view(rows, rec, R)
    rv = s["rv"].double().view(rows, rec, R)
    state = s["state"].double()
    S = state[s["state_slots"]] if decode else torch.zeros(n, rec, R, R, dtype=torch.float64, device="cuda")
    right = torch.empty(rows, rec, R, dtype=torch.float64, device="cuda")
    starts = np.arange(n) if decode else np.concatenate([[0], np.cumsum(lens)[:-1]])
    counts = np.ones(n, dtype=np.int64) if decode else lens
    for t in range(int(counts.max())):
        live = np.flatnonzero(counts > t)
        row, which = torch.from_numpy(starts[live] + t).cuda(), torch.from_numpy(live).cuda()
        new = f[row].unsqueeze(-1) * S[which] + (1 - f[row]).unsqueeze(-1) * rv[row].unsqueeze(-2)
        S[which] = new
        right[row] = torch.einsum("bhkv,bhk->bhv", new, rq[row])
    state[s["state_slots"]] = S
    right = right / torch.sqrt(right.pow(2).mean(-1, keepdim=True) + s["eps"]) * s["norm"].double()
    return [left, right.flatten(1), state, None, None]


def _work_mixer(case):
    lens, z = _lengths(case), MIXERS[case["width"]]
    H, G, D, rec, R, W = z["H"], z["G"], z["D"], z["rec"], z["R"], z["window"]
    decode, over = case["stage"] == "decode", np.maximum(lens - z["window"], 0)
    rows = len(lens) if decode else int(lens.sum())
    keys = int(np.minimum(lens, W).sum()) if decode else rows
    pairs = keys if decode else int((lens * (lens + 1) // 2 - over * (over + 1) // 2).sum())
    state = len(lens) * rec * R * R * 4 * (2 if decode else 1)
    return {"bytes": rows * (3 * H * D + 4 * G * D + 4 * rec * R) * 2 + (keys * 2 * G * D * 2 if decode else 0) + state,
            "flops": pairs * H * (4 * D + 2 * H) + rows * rec * R * R * 5}


def _draw_mixer(rng):
    width = rng.choice([1024, 2048, 4096])
    if rng.random() < 0.5:
        hi = _log(rng, 64, 4096)
        size = dict(stage="decode", seqs=_log(rng, 1, 128))
    else:
        hi = _log(rng, 32, 2048)
        size = dict(stage="prompts", seqs=max(1, min(64, _log(rng, 64, 8192) // hi)))
    return dict(kind="nabalix_mixer", width=width, spread="uniform", lo=max(1, hi // rng.choice([1, 4])), hi=hi, mix=rng.randrange(1 << 20), **size)


# ------------------------------------------------------------------------------------------------ the Taminex delta rule
# Convolution, gated delta rule, norm and output gate of a layer between its two projections; prompts or a decode step.
DELTAS = {1024: dict(H=8, G=4, D=64), 2048: dict(H=16, G=8, D=128), 4096: dict(H=32, G=16, D=128)}
TAPS = 4


def _prepare_delta(case, seed):
    d, lens, z = _Draw(seed), _lengths(case), DELTAS[case["width"]]
    H, G, D, n, decode = z["H"], z["G"], z["D"], len(lens), case["stage"] == "decode"
    rows, width = n if decode else int(lens.sum()), (2 * G + H) * D
    f32 = dict(dtype=torch.float32)
    rule = ops.DeltaRule(H, G, D, D, (0, G * D, 2 * G * D), d.normal(TAPS, width, std=TAPS ** -0.5, **f32), d.normal(H, mean=-1.5, **f32),
                         d.normal(H, mean=-1.5, std=1.5, **f32), d.normal(D, mean=1.0, std=0.1, **f32), 1e-5)
    proj = d.normal(rows, width + H * D + 2 * H)
    gate, b, a = proj[:, width:].split([H * D, H, H], 1)
    s = dict(rule=rule, proj=proj, b=b, a=a, gate=gate, state=d.normal(n + 2, H, D, D, std=0.1, **f32),
             ring=d.normal(n + 2, TAPS, width, **f32), slots=d.ints(d.order.permutation(n + 2)[:n], torch.int64))
    if decode:
        s["lens"] = d.ints(lens, torch.int64)
    else:
        s["cu"] = d.offsets(lens)
    return s


def _run_delta(s):
    if "lens" in s:
        o = ops.delta_step(s["rule"], s["proj"], s["b"], s["a"], s["gate"], s["state"], s["ring"], s["slots"], s["lens"])
    else:
        o = ops.delta_rule(s["rule"], s["proj"], s["b"], s["a"], s["gate"], s["state"], s["ring"], s["slots"], s["cu"], s["cu"])
    return [o, s["state"], s["ring"]]


def _exact_delta(case, seed):
    s, z, lens = _prepare_delta(case, seed), DELTAS[case["width"]], _lengths(case)
    H, G, D, n, decode, c = z["H"], z["G"], z["D"], len(lens), case["stage"] == "decode", s["rule"]
    rows, width = s["proj"].shape[0], c.width
    x, w, ring = s["proj"][:, :width].double(), c.conv_w.double(), s["ring"].double()
    act = x * w[-1]
    starts = np.arange(n) if decode else np.concatenate([[0], np.cumsum(lens)[:-1]])
    counts = np.ones(n, dtype=np.int64) if decode else lens
    for i in range(n):
        slot, at, m = int(s["slots"][i]), int(starts[i]), int(counts[i])
        for back in range(1, TAPS):
            if decode:                     # the input of position p waits in row p mod TAPS
                if lens[i] - 1 >= back:
                    act[at] += w[-1 - back] * ring[slot, (int(lens[i]) - 1 - back) % TAPS]
            elif m > back:
                act[at + back:at + m] += w[-1 - back] * x[at:at + m - back]
        # a portion leaves its last TAPS - 1 inputs behind, a single token itself
        for p in [int(lens[i]) - 1] if decode else range(max(0, m - TAPS + 1), m):
            ring[slot, p % TAPS] = x[at + (0 if decode else p)]
    act = torch.nn.functional.silu(act)
    q, k, v = act.split([G * D, G * D, H * D], 1)
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    of = torch.arange(H, device="cuda") // (H // G)
    q, k, v = unit(q.view(rows, G, D))[:, of] * D ** -0.5, unit(k.view(rows, G, D))[:, of], v.view(rows, H, D)
    beta = torch.sigmoid(s["b"].double())
    g = torch.exp(-torch.exp(c.a_log.double()) * torch.nn.functional.softplus(s["a"].double() + c.dt_bias.double(), threshold=1e9))
    state = s["state"].double()
    fresh = torch.from_numpy(np.asarray(lens - counts == 0)).cuda()
    S = torch.where(fresh[:, None, None, None], torch.zeros((), dtype=torch.float64, device="cuda"), state[s["slots"]])
    o = torch.empty(rows, H, D, dtype=torch.float64, device="cuda")
    for t in range(int(counts.max())):
        live = np.flatnonzero(counts > t)
        row, which = torch.from_numpy(starts[live] + t).cuda(), torch.from_numpy(live).cuda()
        new = g[row][..., None, None] * S[which]
        u = beta[row].unsqueeze(-1) * (v[row] - torch.einsum("bhkv,bhk->bhv", new, k[row]))
        new = new + k[row].unsqueeze(-1) * u.unsqueeze(-2)
        S[which] = new
        o[row] = torch.einsum("bhkv,bhk->bhv", new, q[row])
    state[s["slots"]] = S
    o = o / torch.sqrt(o.pow(2).mean(-1, keepdim=True) + c.eps) * c.norm_w.double()
    return [o.flatten(1) * torch.nn.functional.silu(s["gate"].double()), state, ring]


def _work_delta(case):
    lens, z = _lengths(case), DELTAS[case["width"]]
    H, G, D, decode = z["H"], z["G"], z["D"], case["stage"] == "decode"
    rows, width = len(lens) if decode else int(lens.sum()), (2 * G + H) * D
    return {"bytes": rows * (width + 2 * H * D + 2 * H) * 2 + len(lens) * (H * D * D + TAPS * width) * 4 * (2 if decode else 1),
            "flops": rows * H * D * D * 7}


def _draw_delta(rng):
    width = rng.choice([1024, 2048, 4096])
    if rng.random() < 0.4:
        hi = _log(rng, 8, 4096)
        size = dict(stage="decode", seqs=_log(rng, 1, 256))
    else:
        hi = _log(rng, 32, 4096)
        size = dict(stage="prompts", seqs=max(1, min(64, _log(rng, 64, 16384) // hi)))
    return dict(kind="taminex_delta", width=width, spread="uniform", lo=max(1, hi // rng.choice([1, 4])), hi=hi, mix=rng.randrange(1 << 20), **size)


# ------------------------------------------------------------------------------------------------ mixture of experts
# Routing, both expert projections with SwiGLU and the shared expert, and the weighted sum, behind the router's logits: the
# launches of the decoder's expert layer, from one decoded token to the largest batches that stay on them.
EXPERTS = {1024: dict(ff=704, E=16, K=2), 2048: dict(ff=1024, E=32, K=4)}


def _prepare_experts(case, seed):
    d, z, T, w = _Draw(seed), EXPERTS[case["width"]], case["tokens"], case["width"]
    E, F = z["E"], z["ff"]
    # levels in a random order per token: no choice of experts hangs on a rounding
    order = torch.rand(T, E, generator=d.gen, device=d.device).argsort(-1)
    weight = lambda n, k: d.uniform(E + 1, n, k, lo=-k ** -0.5, hi=k ** -0.5, dtype=torch.bfloat16)
    bias = lambda n, k: d.uniform(E + 1, n, lo=-k ** -0.5, hi=k ** -0.5, dtype=torch.bfloat16)
    return dict(x=d.normal(T, w), logits=((order - E // 2).float() / 8).bfloat16(), bias=torch.zeros(E, device="cuda"), K=z["K"],
                w_in=weight(2 * F, w), b_in=bias(2 * F, w), w_out=weight(w, F), b_out=bias(w, F))


def _run_experts(s):
    x, T = s["x"], s["x"].shape[0]
    tok, experts, weights, ends, place = ops.moe_route(s["logits"], s["bias"], s["K"], identity_tail=True)
    rows = x.index_select(0, tok)
    act = ops.moe_grouped_gemm(rows, s["w_in"], ends, s["b_in"], swiglu=True, dense_rows=T, early_launch=True)
    y = ops.moe_grouped_gemm(act, s["w_out"], ends, s["b_out"], dense_rows=T, early_launch=True)
    return ops.moe_combine(y[:T * s["K"]], None, experts, weights, place, y[T * s["K"]:])


def _expert_sum(x, logits, K, w_in, b_in, w_out, b_out):
    """The layer in 64 bits: routed experts weighted by their renormalised sigmoid scores, then the shared one (the last)."""
    E, F = logits.shape[1], w_out.shape[2]
    one = lambda h, e: torch.nn.functional.silu(h[:, :F]) * h[:, F:] @ w_out[e].double().t() + b_out[e].double()
    run = lambda rows, e: one(rows @ w_in[e].double().t() + b_in[e].double(), e)
    chosen = logits.topk(K, -1).indices
    weights = torch.sigmoid(logits.double()).gather(-1, chosen)
    weights = weights / (weights.sum(-1, keepdim=True) + 1e-10) if K > 1 else weights
    out = run(x, E)
    for e in range(E):
        row, k = (chosen == e).nonzero(as_tuple=True)
        out[row] += weights[row, k].unsqueeze(-1) * run(x[row], e)
    return out


def _exact_experts(case, seed):
    s = _prepare_experts(case, seed)
    return _expert_sum(s["x"].double(), s["logits"], s["K"], s["w_in"], s["b_in"], s["w_out"], s["b_out"])


def _work_experts(case):
    z, T, w = EXPERTS[case["width"]], case["tokens"], case["width"]
    used = min(z["E"], T * z["K"]) + 1
    return {"bytes": used * 3 * w * z["ff"] * 2 + T * (2 * w + z["E"]) * 2, "flops": T * (z["K"] + 1) * 6 * w * z["ff"]}


def _draw_experts(rng):
    return dict(kind="experts", width=rng.choice([1024, 2048]), tokens=_log(rng, 1, 2048))


# ------------------------------------------------------------------------------------------------ a decode step of the engine
# The GQA + MoE decoder with running sequences, one token each, through scheduler bookkeeping, cache pool and captured graph;
# logits instead of sampled tokens.
VOCAB = 32000


def _decoder(case):
    return dict(vocab_size=VOCAB, context_length=2048, d_model=1024, num_layers=case["layers"], num_heads=16, num_kv_heads=4, d_ff=704,
                attention_type="GQA", use_moe=True, moe_layers=list(range(case["layers"])), n_routed_experts=16, num_experts_per_tok=2,
                n_shared_experts=1)


def _decoder_weights(case, seed):
    """Parameters under the decoder's checkpoint names, as torch initialises its layers, norms at one."""
    d, w, width, ff, kv = _Draw(seed), {}, 1024, 704, 256

    def lin(name, n, k):
        w[name + ".weight"], w[name + ".bias"] = d.uniform(n, k, lo=-k ** -0.5, hi=k ** -0.5), d.uniform(n, lo=-k ** -0.5, hi=k ** -0.5)

    def mlp(name):
        lin(name + ".w1", ff, width)
        lin(name + ".w3", ff, width)
        lin(name + ".w2", width, ff)

    ones = lambda n: torch.ones(n, device=d.device)
    w["token_embeddings.weight"] = d.normal(VOCAB, width, dtype=torch.float32)
    for i in range(case["layers"]):
        a, f = f"layers.{i}.att", f"layers.{i}.ffn"
        for name, n in (("q_proj", width), ("k_proj", kv), ("v_proj", kv), ("output_proj", width)):
            lin(f"{a}.{name}", n, width)
        w[a + ".q_norm.weight"], w[a + ".k_norm.weight"] = ones(width), ones(kv)
        for e in range(16):
            mlp(f"{f}.experts.{e}")
        mlp(f + ".shared_expert")
        w[f + ".gate.weight"], w[f + ".gate.expert_bias"] = d.uniform(16, width, lo=-width ** -0.5, hi=width ** -0.5), torch.zeros(16, device=d.device)
        w[f"layers.{i}.att_norm.weight"], w[f"layers.{i}.ffn_norm.weight"] = ones(width), ones(width)
    w["final_norm.weight"] = ones(width)
    lin("lm_head", VOCAB, width)
    return w


def _token_ids(case, seed):
    rng = np.random.default_rng([seed, 7])
    return [rng.integers(0, VOCAB, size=int(n)).tolist() for n in _lengths(case)]


def _prepare_engine(case, seed):
    from llm_from_scratch_b200.engine import SamplingParams
    from llm_from_scratch_b200.engine.llm_engine import LLMEngine
    prompts = _token_ids(case, seed)
    # prompts run eagerly here: capturing their steps would be most of the preparation
    eng = LLMEngine(dict(model=_decoder(case), weights=_decoder_weights(case, seed), dtype="bfloat16", block_size=16, prefill_graphs=False,
                         max_num_sequences=case["seqs"], max_num_batched_tokens=8192, max_model_length=2048, eos=-1, device="cuda:0",
                         max_cached_blocks=sum(len(p) // 16 + 2 for p in prompts) + 8))
    for p in prompts:
        eng.add_request(p, SamplingParams(temperature=0.0, max_tokens=64, ignore_eos=True))
    seqs, runner = [], eng.model_runner
    while len(seqs) < len(prompts):
        batch, _ = eng.scheduler.schedule()
        runner.run(batch, True)
        seqs += batch
    # the last token of every prompt is the one to decode: its keys and values are written again, the same ones
    order = {s.seq_id: i for i, s in enumerate(seqs)}
    return dict(engine=eng, seqs=[seqs[order[i]] for i in sorted(order)], want=[[0]] * len(seqs))


def _run_engine(s):
    return s["engine"].model_runner.run_wanted(s["seqs"], False, s["want"])


def _exact_engine(case, seed):
    w, width = _decoder_weights(case, seed), 1024
    prompts = _token_ids(case, seed)
    lens = [len(p) for p in prompts]
    low = lambda name: w[name].bfloat16().double()            # the engine's matrices are bf16
    lin = lambda x, name: x @ low(name + ".weight").t() + low(name + ".bias")
    rms = lambda x, eps: x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps)
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    ang = pos[:, None].double() * 10000.0 ** (-torch.arange(0, 64, 2, device="cuda").double() / 64)
    cos, sin = ang.cos().unsqueeze(1), ang.sin().unsqueeze(1)

    def turn(x):
        a, b = x.chunk(2, -1)
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    x = w["token_embeddings.weight"][torch.tensor(sum(prompts, []), device="cuda")].double()
    eps = float(torch.finfo(torch.float32).eps)
    for i in range(case["layers"]):
        a, f = f"layers.{i}.att.", f"layers.{i}.ffn."
        h = rms(x, 1e-5)
        q = turn(rms(lin(h, a + "q_proj"), eps).view(-1, 16, 64))
        k = turn(rms(lin(h, a + "k_proj"), eps).view(-1, 4, 64))
        v = lin(h, a + "v_proj").view(-1, 4, 64)
        o = torch.cat([_attend(*part, 64 ** -0.5, 0) for part in zip(q.split(lens), k.split(lens), v.split(lens))])
        x = x + lin(o.flatten(1), a + "output_proj")
        h = rms(x, 1e-5)
        names = [f"{f}experts.{e}." for e in range(16)] + [f + "shared_expert."]
        stack = lambda kind, *parts: torch.stack([torch.cat([w[n + p + kind].bfloat16() for p in parts]) for n in names])
        x = x + _expert_sum(h, h @ low(f + "gate.weight").t(), 2, stack(".weight", "w1", "w3"), stack(".bias", "w1", "w3"),
                            stack(".weight", "w2"), stack(".bias", "w2"))
    last = torch.tensor(np.cumsum(lens) - 1, device="cuda")
    return lin(rms(x[last], 1e-5), "lm_head")


def _work_engine(case):
    lens, n, L, d = _lengths(case), case["seqs"], case["layers"], 1024
    experts = min(16, 2 * n) + 1
    per_layer = (2 * d * d + 2 * d * 256 + 16 * d + experts * 3 * d * 704) * 2
    keys = int(lens.sum()) * 2 * 256 * 2
    active = 2 * d * d + 2 * d * 256 + 16 * d + 3 * 3 * d * 704
    return {"bytes": L * (per_layer + keys) + VOCAB * d * 2 + n * VOCAB * 4,
            "flops": n * 2 * (L * active + VOCAB * d) + L * int(lens.sum()) * 4 * d}


def _draw_engine(rng):
    hi = _log(rng, 32, 1024)
    return dict(kind="engine_step", layers=rng.choice([4, 8, 16]), seqs=_log(rng, 1, 128), spread="uniform", lo=max(2, hi // rng.choice([1, 4, 16])),
                hi=hi, mix=rng.randrange(1 << 20))


# ------------------------------------------------------------------------------------------------ the cases
def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# kind -> (prepare, run, exact, work, draw)
KINDS = {
    "decode": (_prepare_decode, _run_decode, _exact_decode, _work_decode, _draw_decode),
    "prompts": (_prepare_prompts, _run_prompts, _exact_prompts, _work_prompts, _draw_prompts),
    "latent_decode": (_prepare_latent, _run_latent, _exact_latent, _work_latent, _draw_latent),
    "nabalix_mixer": (_prepare_mixer, _run_mixer, _exact_mixer, _work_mixer, _draw_mixer),
    "taminex_delta": (_prepare_delta, _run_delta, _exact_delta, _work_delta, _draw_delta),
    "experts": (_prepare_experts, _run_experts, _exact_experts, _work_experts, _draw_experts),
    "engine_step": (_prepare_engine, _run_engine, _exact_engine, _work_engine, _draw_engine),
}


def listed() -> list[dict]:
    small, large = dict(heads=16, kv_heads=4, dim=64), dict(heads=32, kv_heads=8, dim=128)
    return [
        # a single user's chat: one token against a short context
        dict(name="decode one", kind="decode", dtype="bf16", **small, page=16, seqs=1, spread="uniform", lo=700, hi=700, mix=0),
        # a full batch with contexts of very different lengths
        dict(name="decode batch", kind="decode", dtype="bf16", **large, page=16, seqs=256, spread="log", lo=128, hi=8192, mix=1),
        # the engine's fp32 mode (checking a model against its bf16 run), an ordinary batch
        dict(name="decode fp32", kind="decode", dtype="f32", **small, page=16, seqs=64, spread="uniform", lo=64, hi=1024, mix=2),
        # a prefill step of the continuous batching job: prompts of 64 to 1024 tokens
        dict(name="prompts", kind="prompts", dtype="bf16", **small, seqs=15, spread="uniform", lo=64, hi=1024, mix=3),
        # long documents beside short ones, the largest batch
        dict(name="prompts long", kind="prompts", dtype="bf16", **large, seqs=64, spread="zipf", total=262144, lo=1, hi=16384, mix=5),
        # a prefill step in fp32
        dict(name="prompts fp32", kind="prompts", dtype="f32", **small, seqs=8, spread="uniform", lo=64, hi=1024, mix=4),
        # decoding of a latent-attention model with long contexts
        dict(name="latent decode", kind="latent_decode", heads=16, page=16, seqs=240, spread="uniform", lo=512, hi=16384, mix=4),
        # a prefill and a decode step of the Nabalix decoder's mixer
        dict(name="mixer prompts", kind="nabalix_mixer", stage="prompts", width=2048, seqs=8, spread="uniform", lo=1024, hi=1024, mix=0),
        dict(name="mixer decode", kind="nabalix_mixer", stage="decode", width=1024, seqs=64, spread="uniform", lo=600, hi=1500, mix=6),
        # a prefill step of the Taminex decoder's recurrent layer
        dict(name="delta prompts", kind="taminex_delta", stage="prompts", width=1024, seqs=8, spread="uniform", lo=700, hi=1300, mix=7),
        # the expert layer of a short prefill step
        dict(name="experts", kind="experts", width=1024, tokens=2000),
        # a decode step of the continuous batching job
        dict(name="engine step", kind="engine_step", layers=16, seqs=64, spread="uniform", lo=64, hi=1024, mix=8),
    ]


def draw(rng) -> dict:
    return KINDS[rng.choice(list(KINDS))][4](rng)


def prepare(case: dict, seed: int):
    return case["kind"], KINDS[case["kind"]][0](case, seed)


def run(state):
    kind, s = state
    return KINDS[kind][1](s)


def exact(case: dict, seed: int):
    return KINDS[case["kind"]][2](case, seed)


def work(case: dict) -> dict:
    return KINDS[case["kind"]][3](case)


def tolerance(case: dict):
    if case.get("dtype") == "f32":
        return {"rel": 1e-5}
    if case["kind"] == "engine_step":        # roundings of 16 layers, and experts whose router scores all but tie change places
        return {"rel": 3e-2, "max": 0.9}
    return {"rel": 1e-2}
