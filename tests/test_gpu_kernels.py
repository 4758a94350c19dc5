"""Parity of the CUDA kernels (through the C ABI) against the CPU oracle on seeded inputs.

Tolerances: fp32 kernels 2e-5 max-abs; bf16 kernels 2e-2 max-abs and 1e-2 mean-relative error
against the fp32 oracle evaluated on the same bf16-rounded inputs.
"""
import numpy as np
import pytest
import torch

from llm_from_scratch_b200.workloads import deal_blocks

pytestmark = pytest.mark.gpu

BF16_MAX_ABS = 2e-2
BF16_MEAN_REL = 1e-2
F32_MAX_ABS = 2e-5


def _ops():
    from llm_from_scratch_b200 import ops
    return ops


def _oracle():
    from oracle import attention
    return attention


def assert_close(got: torch.Tensor, want: torch.Tensor, dtype):
    got = got.float().cpu()
    want = want.float().cpu()
    assert torch.isfinite(got).all()
    err = (got - want).abs()
    if dtype == torch.float32:
        assert err.max().item() <= F32_MAX_ABS, err.max().item()
    else:
        assert err.max().item() <= BF16_MAX_ABS, err.max().item()
        rel = err.sum().item() / max(want.abs().sum().item(), 1e-30)
        assert rel <= BF16_MEAN_REL, rel


def _randn(shape, seed, dtype):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(shape, generator=g).to(dtype)


# ----------------------------------------------------------------------------- store_kvcache
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,Hkv,D,bs", [(1, 1, 32, 16), (37, 4, 32, 16), (300, 8, 128, 16),
                                        (64, 4, 64, 256), (5, 3, 20, 4)])
def test_store_kvcache_bit_exact(dtype, T, Hkv, D, bs):
    ops, orc = _ops(), _oracle()
    nb = (T + bs - 1) // bs + 3
    k, v = _randn((T, Hkv, D), 1, dtype), _randn((T, Hkv, D), 2, dtype)
    rng = np.random.default_rng(2)
    slots = torch.from_numpy(rng.permutation(nb * bs)[:T].astype(np.int64))
    if T > 3:
        slots[1] = -1  # graph-replay padding
    kc0, vc0 = _randn((nb, bs, Hkv, D), 3, dtype), _randn((nb, bs, Hkv, D), 4, dtype)
    kc_ref, vc_ref = kc0.clone(), vc0.clone()
    orc.store_kvcache(k, v, kc_ref, vc_ref, slots)
    kc, vc = kc0.cuda(), vc0.cuda()
    ops.store_kvcache(k.cuda(), v.cuda(), kc, vc, slots.cuda())
    ops.check_status()
    assert torch.equal(kc.cpu(), kc_ref) and torch.equal(vc.cpu(), vc_ref)


def test_store_kvcache_strided_views_of_fused_qkv():
    ops, orc = _ops(), _oracle()
    T, Hq, Hkv, D, bs, nb = 50, 8, 2, 64, 16, 8
    qkv = _randn((T, (Hq + 2 * Hkv) * D), 5, torch.bfloat16)
    k = qkv[:, Hq * D:(Hq + Hkv) * D].view(T, Hkv, D)
    v = qkv[:, (Hq + Hkv) * D:].view(T, Hkv, D)
    slots = torch.from_numpy(np.random.default_rng(0).permutation(nb * bs)[:T].astype(np.int64))
    kc_ref, vc_ref = torch.zeros(nb, bs, Hkv, D, dtype=torch.bfloat16), torch.zeros(nb, bs, Hkv, D, dtype=torch.bfloat16)
    orc.store_kvcache(k, v, kc_ref, vc_ref, slots)
    qkv_d = qkv.cuda()
    kd = qkv_d[:, Hq * D:(Hq + Hkv) * D].view(T, Hkv, D)
    vd = qkv_d[:, (Hq + Hkv) * D:].view(T, Hkv, D)
    kc, vc = torch.zeros_like(kc_ref).cuda(), torch.zeros_like(vc_ref).cuda()
    ops.store_kvcache(kd, vd, kc, vc, slots.cuda())
    assert torch.equal(kc.cpu(), kc_ref) and torch.equal(vc.cpu(), vc_ref)


def test_store_kvcache_out_of_pool_slot_is_skipped_and_reported():
    ops = _ops()
    from llm_from_scratch_b200._lib import B200Error
    k = _randn((4, 2, 32), 1, torch.bfloat16).cuda()
    kc = torch.zeros(2, 16, 2, 32, dtype=torch.bfloat16, device="cuda")
    vc = torch.zeros_like(kc)
    slots = torch.tensor([0, 1, 2, 10 ** 9], dtype=torch.int64, device="cuda")
    ops.store_kvcache(k, k, kc, vc, slots)
    with pytest.raises(B200Error):
        ops.check_status()
    ops.check_status()  # cleared by the read
    assert torch.equal(kc.view(-1, 2, 32)[:3], k[:3])


def test_store_kvcache_round_trip_full_size():
    """Size-independent property at the ragged-prefill stress size: scatter through a shuffled
    slot mapping, gather back through the same mapping, bit-identical."""
    ops = _ops()
    T, Hkv, D, bs = 262144, 8, 128, 16
    g = torch.Generator(device="cuda").manual_seed(2)
    k = torch.randn(T, Hkv, D, generator=g, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(T, Hkv, D, generator=g, device="cuda", dtype=torch.bfloat16)
    slots = torch.randperm(T, generator=g, device="cuda")
    kc = torch.zeros(T // bs, bs, Hkv, D, dtype=torch.bfloat16, device="cuda")
    vc = torch.zeros_like(kc)
    ops.store_kvcache(k, v, kc, vc, slots)
    ops.check_status()
    assert torch.equal(kc.view(T, Hkv, D)[slots], k)
    assert torch.equal(vc.view(T, Hkv, D)[slots], v)


# ----------------------------------------------------------------------------- paged decode
def _decode_case(lens, Hq, Hkv, D, bs, dtype, seed=0, pad_value=-1):
    rng = np.random.default_rng(seed)
    case = deal_blocks(lens, bs, rng, pad_blocks=2, pad_value=pad_value)
    B = len(lens)
    q = _randn((B, Hq, D), seed + 10, dtype)
    kc = _randn((case.num_blocks, bs, Hkv, D), seed + 11, dtype)
    vc = _randn((case.num_blocks, bs, Hkv, D), seed + 12, dtype)
    return case, q, kc, vc


def _run_decode(case, q, kc, vc, scale):
    ops = _ops()
    bt = torch.from_numpy(case.block_tables).cuda()
    cl = torch.from_numpy(case.context_lens).cuda()
    out = ops.paged_decode_gqa(q.cuda(), kc.cuda(), vc.cuda(), bt, cl, scale)
    ops.check_status()
    return out


@pytest.mark.parametrize("Hq,Hkv,D", [(32, 8, 128), (16, 4, 64), (16, 4, 32), (8, 8, 128),
                                      (16, 2, 64), (16, 1, 128), (32, 2, 128), (12, 4, 64)])
def test_paged_decode_bf16_matches_oracle(Hq, Hkv, D):
    lens = [1, 15, 16, 17, 31, 32, 33, 100, 0, 257, 1000, 64, 5, 2049]
    case, q, kc, vc = _decode_case(lens, Hq, Hkv, D, 16, torch.bfloat16, seed=Hq + D)
    scale = D ** -0.5
    want = _oracle().paged_decode_gqa(q, kc, vc, case.block_tables, case.context_lens, scale)
    got = _run_decode(case, q, kc, vc, scale)
    assert_close(got, want, torch.bfloat16)
    assert (got[8] == 0).all()  # empty context -> zero row


def test_paged_decode_bf16_long_sequence_split_across_ctas():
    lens = [6000, 3, 16 * 148 + 7, 129]
    case, q, kc, vc = _decode_case(lens, 32, 8, 128, 16, torch.bfloat16, seed=7)
    scale = 128 ** -0.5
    want = _oracle().paged_decode_gqa(q, kc, vc, case.block_tables, case.context_lens, scale)
    got = _run_decode(case, q, kc, vc, scale)
    assert_close(got, want, torch.bfloat16)


@pytest.mark.parametrize("Hq,Hkv,D,bs", [(32, 8, 128, 64), (12, 1, 128, 256), (6, 3, 128, 16), (16, 1, 128, 32)])
@pytest.mark.parametrize("lens", [[1], [700], [16, 64, 65, 128, 129], [511, 0, 513, 2048, 15], [1030] * 40])
@pytest.mark.parametrize("sink", [False, True])
def test_decode_in_clusters_and_in_one_stream(Hq, Hkv, D, bs, lens, sink):
    """Both bf16 forms on the same contexts: block tables as wide as the contexts need go to clusters of CTAs, tables that allow
    far longer contexts to the streaming kernel.  Contexts around the blocks, warps and CTAs that share them; empty ones;
    block numbers behind a context are never read."""
    ops, orc = _ops(), _oracle()
    case, q, kc, vc = _decode_case(lens, Hq, Hkv, D, bs, torch.bfloat16, seed=D + len(lens))
    s = _randn((Hq,), 5, torch.float32) if sink else None
    want = orc.paged_decode_gqa(q, kc, vc, case.block_tables, case.context_lens, D ** -0.5)
    if sink:        # the sum of a row is that of its weights without sinks
        scores = [torch.einsum("hd,nhd->hn", q[i].float(), kc[torch.from_numpy(case.block_tables[i, :-(-n // bs)]).long()].flatten(0, 1)[:n]
                               .float().repeat_interleave(Hq // Hkv, 1)) * D ** -0.5 for i, n in enumerate(lens)]
        lse = torch.stack([torch.logsumexp(x, -1) if x.shape[1] else torch.full((Hq,), float("inf")) for x in scores])
        want = want * torch.sigmoid(lse - s)[:, :, None]
    wide = np.full((len(lens), 8 * 4096 // bs * 2 + 8), 2 ** 30, dtype=np.int32)
    wide[:, :case.block_tables.shape[1]] = case.block_tables
    for table in (case.block_tables, wide):
        got = ops.paged_decode_gqa(q.cuda(), kc.cuda(), vc.cuda(), torch.from_numpy(table).cuda(),
                                   torch.from_numpy(case.context_lens).cuda(), D ** -0.5, sink=None if s is None else s.cuda())
        ops.check_status()
        assert_close(got, want, torch.bfloat16)


@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 128), (torch.float32, 32), (torch.float32, 64), (torch.float32, 80), (torch.float32, 128)])
@pytest.mark.parametrize("gone", [(16, 32), (0, 16), (0, 8), (64, 128), (100, 164), (1, 300), (0, 299)])
def test_decode_of_keys_whose_scores_are_minus_infinity(dtype, D, gone):
    """They weigh nothing, also where a block, a trip of a lane, a warp or a whole CTA of a cluster holds no others."""
    ops, orc = _ops(), _oracle()
    case, q, kc, vc = _decode_case([300], 8, 2, D, 16, dtype, seed=D)
    q[..., 0] = 1
    rows = torch.from_numpy(case.block_tables[0, :19]).long()[:, None] * 16 + torch.arange(16)
    rows = rows.flatten()[:300]
    left = torch.tensor([i for i in range(300) if not gone[0] <= i < gone[1]])
    k, v = kc.flatten(0, 1)[rows[left]], vc.flatten(0, 1)[rows[left]]
    kc.view(-1, 2, D)[rows[gone[0]:gone[1]], :, 0] = float("-inf")
    p = torch.softmax(torch.einsum("hd,nhd->hn", q[0].double(), k.double().repeat_interleave(4, 1)) * D ** -0.5, -1)
    want = torch.einsum("hn,nhd->hd", p, v.double().repeat_interleave(4, 1))[None]
    got = ops.paged_decode_gqa(q.cuda(), kc.cuda(), vc.cuda(), torch.from_numpy(case.block_tables).cuda(),
                               torch.from_numpy(case.context_lens).cuda(), D ** -0.5)
    ops.check_status()
    assert_close(got, want, dtype)


@pytest.mark.parametrize("dtype,D,page", [(torch.float32, 32, 16), (torch.float32, 64, 16), (torch.float32, 128, 16), (torch.float32, 80, 16),
                                          (torch.bfloat16, 128, 16), (torch.bfloat16, 64, 16), (torch.bfloat16, 64, 5)])
@pytest.mark.parametrize("n,at", [(300, 0), (300, 170), (1, 0)])
def test_a_broken_key_row_is_seen_in_the_output(dtype, D, page, n, at):
    """A NaN in one visible key makes the rows of its query heads NaN, not zeros, and no others."""
    ops = _ops()
    case, q, kc, vc = _decode_case([n], 8, 2, D, page, dtype, seed=D)
    kc[case.block_tables[0, at // page], at % page, 1, 3] = float("nan")
    got = _run_decode(case, q, kc, vc, D ** -0.5)
    assert torch.isfinite(got[0, :4]).all() and torch.isnan(got[0, 4:]).all()


@pytest.mark.parametrize("latent", [False, True])
def test_merge_of_one_long_context_in_a_large_batch(latent):
    """The merge's CTAs take several columns each where there are many, and the long context has more pieces than fit their shared
    memory at a time; empty contexts are zeros."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    lens = [64] * (240 if latent else 1024)
    lens[7], lens[3], lens[-1] = 9000, 0, 33
    case = deal_blocks(lens, 16, np.random.default_rng(3), pad_blocks=1)
    tables, ctx = torch.from_numpy(case.block_tables).cuda(), torch.from_numpy(case.context_lens).cuda()
    if latent:
        H, cache, qa, qr = 32, r(case.num_blocks, 16, 576), r(len(lens), 32, 512), r(len(lens), 32, 64)
        got = ops.mla_decode(qa, qr, cache, tables, ctx, 0.07)
    else:
        H, q, kc, vc = 64, r(len(lens), 64, 64), r(case.num_blocks, 16, 8, 64), r(case.num_blocks, 16, 8, 64)
        got = ops.paged_decode_gqa(q, kc, vc, tables, ctx, 0.125)
    ops.check_status()
    assert (got[3] == 0).all()
    for i in (0, 6, 7, 8, len(lens) - 1):
        rows = (tables[i, :-(-lens[i] // 16)].long()[:, None] * 16 + torch.arange(16, device="cuda")).flatten()[:lens[i]]
        if latent:
            keys = cache.view(-1, 576)[rows].double()
            want = torch.softmax((qa[i].double() @ keys[:, :512].T + qr[i].double() @ keys[:, 512:].T) * 0.07, -1) @ keys[:, :512]
        else:
            k, v = (c.view(-1, 8, 64)[rows].double().repeat_interleave(8, 1) for c in (kc, vc))
            want = torch.einsum("hn,nhd->hd", torch.softmax(torch.einsum("hd,nhd->hn", q[i].double(), k) * 0.125, -1), v)
        assert_close(got[i], want, torch.bfloat16)


def test_paged_decode_bf16_single_short_sequence_and_stale_table_entries():
    # entries past ceil(len/16) hold stale ids outside the pool: they must never be read
    case, q, kc, vc = _decode_case([20], 32, 8, 128, 16, torch.bfloat16, seed=3)
    bt = np.full((1, 40), 2 ** 30, dtype=np.int32)
    bt[0, :2] = case.block_tables[0, :2]
    case.block_tables = bt
    scale = 128 ** -0.5
    want = _oracle().paged_decode_gqa(q, kc, vc, case.block_tables, case.context_lens, scale)
    got = _run_decode(case, q, kc, vc, scale)
    assert_close(got, want, torch.bfloat16)


def test_paged_decode_rejects_block_id_outside_pool_without_reading_it():
    from llm_from_scratch_b200._lib import B200Error
    ops = _ops()
    case, q, kc, vc = _decode_case([40, 40], 32, 8, 128, 16, torch.bfloat16, seed=4)
    case.block_tables[1, 1] = case.num_blocks + 5
    bt = torch.from_numpy(case.block_tables).cuda()
    cl = torch.from_numpy(case.context_lens).cuda()
    ops.paged_decode_gqa(q.cuda(), kc.cuda(), vc.cuda(), bt, cl, 128 ** -0.5)
    with pytest.raises(B200Error):
        ops.check_status()


def test_paged_decode_is_deterministic_and_repeatable():
    case, q, kc, vc = _decode_case([700, 33, 1500, 90, 4000], 32, 8, 128, 16, torch.bfloat16, seed=5)
    a = _run_decode(case, q, kc, vc, 128 ** -0.5)
    b = _run_decode(case, q, kc, vc, 128 ** -0.5)
    assert torch.equal(a, b)


@pytest.mark.parametrize("Hq,Hkv,D,bs", [(16, 4, 32, 16), (8, 2, 48, 8), (4, 4, 128, 256)])
def test_paged_decode_fp32_matches_oracle(Hq, Hkv, D, bs):
    lens = [1, bs, bs + 1, 0, 77, 300]
    case, q, kc, vc = _decode_case(lens, Hq, Hkv, D, bs, torch.float32, seed=D)
    scale = D ** -0.5
    want = _oracle().paged_decode_gqa(q, kc, vc, case.block_tables, case.context_lens, scale)
    got = _run_decode(case, q, kc, vc, scale)
    assert_close(got, want, torch.float32)


def test_paged_decode_bf16_generic_path_for_other_block_sizes():
    case, q, kc, vc = _decode_case([5, 300, 64], 8, 2, 64, 32, torch.bfloat16, seed=9)
    want = _oracle().paged_decode_gqa(q, kc, vc, case.block_tables, case.context_lens, 0.125)
    got = _run_decode(case, q, kc, vc, 0.125)
    assert_close(got, want, torch.bfloat16)


def test_paged_decode_microbenchmark_shape_sampled_rows():
    """Benchmark-size batch (256 sequences, log-uniform contexts up to 8192); the oracle checks a
    sample of rows, and decoding each sampled row alone must give the same bits as in the batch
    only up to split placement, so the comparison is by tolerance."""
    from llm_from_scratch_b200.workloads import c2_decode_case
    ops = _ops()
    case = c2_decode_case()
    Hq, Hkv, D = 32, 8, 128
    g = torch.Generator(device="cuda").manual_seed(1)
    kc = torch.randn(case.num_blocks, 16, Hkv, D, generator=g, device="cuda", dtype=torch.bfloat16)
    vc = torch.randn(case.num_blocks, 16, Hkv, D, generator=g, device="cuda", dtype=torch.bfloat16)
    q = torch.randn(case.batch, Hq, D, generator=g, device="cuda", dtype=torch.bfloat16)
    bt = torch.from_numpy(case.block_tables).cuda()
    cl = torch.from_numpy(case.context_lens).cuda()
    out = ops.paged_decode_gqa(q, kc, vc, bt, cl, D ** -0.5)
    ops.check_status()
    assert torch.isfinite(out.float()).all()
    rows = [0, 1, 17, 100, 255, int(np.argmax(case.context_lens)), int(np.argmin(case.context_lens))]
    for b in rows:
        L = int(case.context_lens[b])
        nblk = (L + 15) // 16
        ids = torch.from_numpy(case.block_tables[b, :nblk].astype(np.int64)).cuda()
        kcb, vcb = kc[ids].cpu(), vc[ids].cpu()
        want = _oracle().paged_decode_gqa(q[b:b + 1].cpu(), kcb, vcb, [list(range(nblk))], [L], D ** -0.5)
        assert_close(out[b:b + 1], want, torch.bfloat16)


# ----------------------------------------------------------------------------- varlen prefill
def _prefill_inputs(lens, Hq, Hkv, Dqk, Dv, dtype, seed):
    T = sum(lens)
    q = _randn((T, Hq, Dqk), seed, dtype)
    k = _randn((T, Hkv, Dqk), seed + 1, dtype)
    v = _randn((T, Hkv, Dv), seed + 2, dtype)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32)
    return q, k, v, cu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("Hq,Hkv,D", [(16, 4, 32), (32, 8, 128), (4, 4, 64), (16, 4, 64)])
def test_prefill_varlen_matches_oracle(dtype, Hq, Hkv, D):
    ops = _ops()
    lens = [1, 16, 17, 45, 128, 3, 200]
    q, k, v, cu = _prefill_inputs(lens, Hq, Hkv, D, D, dtype, seed=D + Hq)
    scale = D ** -0.5
    want = _oracle().prefill_varlen(q, k, v, cu, cu, scale)
    got = ops.prefill_varlen(q.cuda(), k.cuda(), v.cuda(), cu.cuda(), cu.cuda(), max(lens), max(lens), scale)
    ops.check_status()
    assert_close(got, want, dtype)


@pytest.mark.parametrize("Hq,Hkv,D", [(16, 4, 64), (32, 8, 128), (4, 4, 32)])
def test_prefill_plan_lists_every_tile_once_and_gives_identical_output(Hq, Hkv, D):
    """The tile list holds every (sequence, tile) pair exactly once, highest tiles first; attention
    launched from it is bit-identical to the (sequence x tile rank) grid, also when cu_seqlens has
    unused trailing sequences and q has padding rows (the fixed-size buffers of a captured step)."""
    ops = _ops()
    lens = [300, 0, 1, 64, 65, 700, 128, 5]
    q, k, v, cu = _prefill_inputs(lens, Hq, Hkv, D, D, torch.bfloat16, seed=77)
    q, k, v, cu = q.cuda(), k.cuda(), v.cuda(), cu.cuda()
    scale = D ** -0.5
    rows = ops.prefill_tile_rows(Hq, Hkv, D, D, torch.bfloat16)
    # tcgen05 row-pair kernel / tcgen05 four-heads-per-CTA kernel (head_dim 64, groups of four) / mma.sync kernel
    assert rows == {128: 256, 64: 128, 32: 64}[D]
    plan = ops.prefill_plan(cu, sum(lens), max(lens), rows)
    ops.check_status()
    buf = plan.buffer.cpu().numpy()
    want_tiles = sorted((s, t) for s, L in enumerate(lens) for t in range((L + rows - 1) // rows))
    assert buf[0] == len(want_tiles) and buf[1] == rows and buf[2] == plan.capacity
    entries = buf[4:4 + buf[0]].astype(np.uint32)
    assert sorted((int(e >> 16), int(e & 0xffff)) for e in entries) == want_tiles
    ranks = (entries & 0xffff).astype(np.int64)
    assert (ranks[1:] <= ranks[:-1]).all()
    base = ops.prefill_varlen(q, k, v, cu, cu, max(lens), max(lens), scale)
    planned = ops.prefill_varlen(q, k, v, cu, cu, max(lens), max(lens), scale, plan=plan)
    ops.check_status()
    assert torch.equal(base, planned)
    # fixed-size buffers: 3 unused sequences, 100 padding rows, bounds instead of exact sizes
    T = sum(lens)
    pad = lambda x: torch.cat([x, torch.zeros(100, *x.shape[1:], dtype=x.dtype, device="cuda")])
    cu_pad = torch.cat([cu, cu[-1:].expand(3)]).contiguous()
    plan2 = ops.prefill_plan(cu_pad, T + 100, T + 100, rows)
    out = torch.zeros(T + 100, Hq, D, dtype=torch.bfloat16, device="cuda")
    ops.prefill_varlen(pad(q), pad(k), pad(v), cu_pad, cu_pad, T + 100, T + 100, scale, out=out, plan=plan2)
    ops.check_status()
    assert torch.equal(out[:T], base) and (out[T:] == 0).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_prefill_varlen_with_cached_prefix_through_block_tables(dtype):
    ops, orc = _ops(), _oracle()
    Hq, Hkv, D, bs = 16, 4, 64, 16
    k_lens = [48, 100, 16, 37]
    cached = [32, 64, 0, 16]
    q_lens = [a - b for a, b in zip(k_lens, cached)]
    rng = np.random.default_rng(3)
    case = deal_blocks(k_lens, bs, rng, pad_blocks=1)
    kc = _randn((case.num_blocks, bs, Hkv, D), 21, dtype)
    vc = _randn((case.num_blocks, bs, Hkv, D), 22, dtype)
    q = _randn((sum(q_lens), Hq, D), 23, dtype)
    cu_q = torch.tensor(np.concatenate([[0], np.cumsum(q_lens)]), dtype=torch.int32)
    cu_k = torch.tensor(np.concatenate([[0], np.cumsum(k_lens)]), dtype=torch.int32)
    scale = D ** -0.5
    want = orc.prefill_varlen(q, None, None, cu_q, cu_k, scale, kc, vc, case.block_tables)
    got = ops.prefill_varlen(q.cuda(), None, None, cu_q.cuda(), cu_k.cuda(), max(q_lens), max(k_lens), scale,
                             kc.cuda(), vc.cuda(), torch.from_numpy(case.block_tables).cuda())
    ops.check_status()
    assert_close(got, want, dtype)


def test_prefill_varlen_head_dim_128_cached_prefix_and_many_tiles():
    """head_dim 128 with an even group size takes the tcgen05 path: packed and paged K/V, lengths
    around the 128-row tile boundaries, several KV tiles per query tile."""
    ops, orc = _ops(), _oracle()
    Hq, Hkv, D, bs = 8, 2, 128, 16
    k_lens = [127, 128, 129, 300, 1, 515, 256]
    cached = [0, 64, 16, 160, 0, 400, 128]
    q_lens = [a - b for a, b in zip(k_lens, cached)]
    case = deal_blocks(k_lens, bs, np.random.default_rng(13), pad_blocks=1)
    kc = _randn((case.num_blocks, bs, Hkv, D), 31, torch.bfloat16)
    vc = _randn((case.num_blocks, bs, Hkv, D), 32, torch.bfloat16)
    q = _randn((sum(q_lens), Hq, D), 33, torch.bfloat16)
    cu_q = torch.tensor(np.concatenate([[0], np.cumsum(q_lens)]), dtype=torch.int32)
    cu_k = torch.tensor(np.concatenate([[0], np.cumsum(k_lens)]), dtype=torch.int32)
    scale = D ** -0.5
    want = orc.prefill_varlen(q, None, None, cu_q, cu_k, scale, kc, vc, case.block_tables)
    got = ops.prefill_varlen(q.cuda(), None, None, cu_q.cuda(), cu_k.cuda(), max(q_lens), max(k_lens), scale,
                             kc.cuda(), vc.cuda(), torch.from_numpy(case.block_tables).cuda())
    ops.check_status()
    assert_close(got, want, torch.bfloat16)
    # scores with a large spread exercise the lazy rescaling of the output accumulator
    lens = [400, 130]
    q2, k2, v2, cu = _prefill_inputs(lens, Hq, Hkv, D, D, torch.bfloat16, seed=91)
    k2 = (k2.float() * torch.linspace(0.2, 6.0, sum(lens)).view(-1, 1, 1)).to(torch.bfloat16)
    want = orc.prefill_varlen(q2, k2, v2, cu, cu, scale)
    got = ops.prefill_varlen(q2.cuda(), k2.cuda(), v2.cuda(), cu.cuda(), cu.cuda(), max(lens), max(lens), scale)
    ops.check_status()
    assert_close(got, want, torch.bfloat16)


def test_prefill_varlen_mla_head_dims_192_128():
    ops = _ops()
    lens = [33, 70, 5]
    q, k, v, cu = _prefill_inputs(lens, 16, 16, 192, 128, torch.bfloat16, seed=40)
    scale = 192 ** -0.5
    want = _oracle().prefill_varlen(q, k, v, cu, cu, scale)
    got = ops.prefill_varlen(q.cuda(), k.cuda(), v.cuda(), cu.cuda(), cu.cuda(), max(lens), max(lens), scale)
    assert_close(got, want, torch.bfloat16)


@pytest.mark.parametrize("Hq,Hkv,Dqk,Dv", [(4, 4, 192, 128), (6, 2, 128, 128), (3, 1, 128, 128)])
def test_prefill_row_pair_kernel_long_ragged_batch(Hq, Hkv, Dqk, Dv):
    """Head shapes served by the tcgen05 kernel that gives a CTA 256 query rows of one head (MLA's
    192/128, head_dim 128 with an odd group size): lengths around the 128- and 256-row
    boundaries, sequences that end inside the first half of a CTA, many key tiles; with and without
    the tile list."""
    ops = _ops()
    lens = [1, 127, 128, 129, 255, 256, 257, 700, 1500, 2, 64, 385]
    q, k, v, cu = _prefill_inputs(lens, Hq, Hkv, Dqk, Dv, torch.bfloat16, seed=Dqk + Hq)
    scale = Dqk ** -0.5
    want = _oracle().prefill_varlen(q, k, v, cu, cu, scale)
    q, k, v, cu = q.cuda(), k.cuda(), v.cuda(), cu.cuda()
    got = ops.prefill_varlen(q, k, v, cu, cu, max(lens), max(lens), scale)
    ops.check_status()
    assert_close(got, want, torch.bfloat16)
    rows = ops.prefill_tile_rows(Hq, Hkv, Dqk, Dv, torch.bfloat16)
    assert rows == 256
    plan = ops.prefill_plan(cu, sum(lens), max(lens), rows)
    planned = ops.prefill_varlen(q, k, v, cu, cu, max(lens), max(lens), scale, plan=plan)
    ops.check_status()
    assert torch.equal(planned, got)


@pytest.mark.parametrize("Hq,Hkv,Dqk,Dv", [(4, 4, 192, 128), (4, 2, 128, 128)])
def test_prefill_row_pair_kernel_scores_that_outgrow_the_reference_maximum(Hq, Hkv, Dqk, Dv):
    """The row-pair kernel rescales its output accumulator lazily: a row's reference maximum moves only when a
    tile's maximum exceeds it by more than 2^8, so probabilities of a tile may be up to 2^8 large before the
    accumulator is rescaled.  Keys whose scores lie far above everything before them (here from position 100 on,
    then again from 900 on) force both the large-probability path and the rescale path, and must still give the
    oracle's result.

    Bound: 2e-2 max-abs where the result is at most 1 in magnitude; above, two bf16 steps of the result's
    magnitude.  With nearly one-hot probabilities an output element is essentially one value element (|v| up to
    4.5 here, bf16 step 2^-5 = 0.031 in [4, 8)): the bf16 rounding of the output alone is up to half a step and
    the rounding of P to bf16 adds up to about one more, which no kernel that returns bf16 can avoid."""
    ops = _ops()
    lens = [1300, 257, 90]
    q, k, v, cu = _prefill_inputs(lens, Hq, Hkv, Dqk, Dv, torch.bfloat16, seed=91)
    pos = torch.cat([torch.arange(n) for n in lens])
    k = (k.float() * torch.where(pos >= 900, 60.0, torch.where(pos >= 100, 25.0, 1.0)).view(-1, 1, 1)).to(torch.bfloat16)
    scale = Dqk ** -0.5
    want = _oracle().prefill_varlen(q, k, v, cu, cu, scale)
    got = ops.prefill_varlen(q.cuda(), k.cuda(), v.cuda(), cu.cuda(), cu.cuda(), max(lens), max(lens), scale)
    ops.check_status()
    assert torch.isfinite(got.float()).all()
    want = want.float()
    err = (got.float().cpu() - want).abs()
    step = torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(1e-30))) - 7)      # bf16 spacing at |want|
    bound = torch.maximum(torch.full_like(want, 2e-2), 2 * step)
    assert (err <= bound).all(), ((err - bound).max().item(), err.max().item())
    assert err.mean().item() <= 3e-3, err.mean().item()


# ----------------------------------------------------------------------------- MLA decode
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,r,dr", [(16, 512, 64), (8, 128, 32), (16, 256, 16)])
def test_mla_decode_matches_oracle(dtype, H, r, dr):
    ops = _ops()
    lens = [1, 16, 17, 0, 100, 513, 40]
    bs = 16
    case = deal_blocks(lens, bs, np.random.default_rng(4), pad_blocks=2)
    B = len(lens)
    qa = (_randn((B, H, r), 50, torch.float32) * 0.3).to(dtype)
    qr = _randn((B, H, dr), 51, dtype)
    lat = _randn((case.num_blocks, bs, r + dr), 52, dtype)
    scale = (128 + dr) ** -0.5
    want = _oracle().mla_decode(qa, qr, lat, case.block_tables, case.context_lens, scale)
    got = ops.mla_decode(qa.cuda(), qr.cuda(), lat.cuda(), torch.from_numpy(case.block_tables).cuda(),
                         torch.from_numpy(case.context_lens).cuda(), scale)
    ops.check_status()
    assert_close(got, want, dtype)


# ----------------------------------------------------------------------------- prefill, larger cases
@pytest.mark.parametrize("Hq,Hkv,D", [(8, 2, 128), (4, 4, 64), (4, 1, 32)])
def test_prefill_varlen_long_ragged_batch_bf16(Hq, Hkv, D):
    ops = _ops()
    lens = [1, 63, 64, 65, 127, 128, 129, 700, 1500, 2]
    q, k, v, cu = _prefill_inputs(lens, Hq, Hkv, D, D, torch.bfloat16, seed=3 * D)
    scale = D ** -0.5
    want = _oracle().prefill_varlen(q, k, v, cu, cu, scale)
    got = ops.prefill_varlen(q.cuda(), k.cuda(), v.cuda(), cu.cuda(), cu.cuda(), max(lens), max(lens), scale)
    ops.check_status()
    assert_close(got, want, torch.bfloat16)


def test_prefill_varlen_strided_q_and_v_views():
    """q/k/v as column slices of one fused projection output (token stride > row width)."""
    ops = _ops()
    lens = [70, 9, 130]
    T, Hq, Hkv, D = sum(lens), 8, 2, 64
    qkv = _randn((T, (Hq + 2 * Hkv) * D), 77, torch.bfloat16)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32)

    def views(t):
        return (t[:, :Hq * D].view(T, Hq, D), t[:, Hq * D:(Hq + Hkv) * D].view(T, Hkv, D),
                t[:, (Hq + Hkv) * D:].view(T, Hkv, D))
    q, k, v = views(qkv)
    want = _oracle().prefill_varlen(q, k, v, cu, cu, D ** -0.5)
    qd, kd, vd = views(qkv.cuda())
    got = ops.prefill_varlen(qd, kd, vd, cu.cuda(), cu.cuda(), max(lens), max(lens), D ** -0.5)
    assert_close(got, want, torch.bfloat16)


def test_prefill_varlen_stress_shape_properties():
    """Ragged prefill stress shape (64 sequences, Zipf(1.2) lengths in [1,16384], 262,144 tokens,
    32/8 heads, head_dim 128): too large for the CPU oracle, so size-independent properties:
    (1) a sequence computed alone gives bit-identical rows to the same sequence inside the batch;
    (2) causality: changing the last third of a sequence's K/V leaves its earlier rows bit-identical;
    (3) the first row of every sequence equals its own V row (softmax over one key)."""
    from llm_from_scratch_b200.workloads import c5_prefill_lengths
    ops = _ops()
    lens = c5_prefill_lengths()
    T, Hq, Hkv, D = int(lens.sum()), 32, 8, 128
    g = torch.Generator(device="cuda").manual_seed(2)
    q = torch.randn(T, Hq, D, generator=g, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(T, Hkv, D, generator=g, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(T, Hkv, D, generator=g, device="cuda", dtype=torch.bfloat16)
    cu_np = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cu = torch.from_numpy(cu_np).cuda()
    scale = D ** -0.5
    out = ops.prefill_varlen(q, k, v, cu, cu, int(lens.max()), int(lens.max()), scale)
    ops.check_status()
    assert torch.isfinite(out.float()).all()
    first_rows = torch.from_numpy(cu_np[:-1].astype(np.int64)).cuda()
    want_first = v[first_rows].repeat_interleave(Hq // Hkv, dim=1)
    assert (out[first_rows].float() - want_first.float()).abs().max().item() <= 1e-2
    order = np.argsort(-lens)
    for s in (int(order[0]), int(order[len(order) // 2]), int(order[-1])):
        a, b = int(cu_np[s]), int(cu_np[s + 1])
        L = b - a
        cu1 = torch.tensor([0, L], dtype=torch.int32, device="cuda")
        alone = ops.prefill_varlen(q[a:b], k[a:b], v[a:b], cu1, cu1, L, L, scale)
        assert torch.equal(alone, out[a:b])
        if L >= 3:
            cut = a + (2 * L) // 3
            k2, v2 = k[a:b].clone(), v[a:b].clone()
            k2[cut - a:] = 0
            v2[cut - a:] = 1
            changed = ops.prefill_varlen(q[a:b], k2, v2, cu1, cu1, L, L, scale)
            assert torch.equal(changed[:cut - a], out[a:cut])


def test_mla_decode_bf16_long_contexts_cut_across_ctas():
    ops = _ops()
    H, r, dr, bs = 16, 512, 64, 16
    lens = [9000, 3, 16 * 148 * 2 + 5, 64, 65, 1]
    case = deal_blocks(lens, bs, np.random.default_rng(8), pad_blocks=2)
    B = len(lens)
    qa = (_randn((B, H, r), 60, torch.float32) * 0.2).to(torch.bfloat16)
    qr = _randn((B, H, dr), 61, torch.bfloat16)
    lat = _randn((case.num_blocks, bs, r + dr), 62, torch.bfloat16)
    scale = 192 ** -0.5
    want = _oracle().mla_decode(qa, qr, lat, case.block_tables, case.context_lens, scale)
    bt, cl = torch.from_numpy(case.block_tables).cuda(), torch.from_numpy(case.context_lens).cuda()
    got = ops.mla_decode(qa.cuda(), qr.cuda(), lat.cuda(), bt, cl, scale)
    ops.check_status()
    assert_close(got, want, torch.bfloat16)
    again = ops.mla_decode(qa.cuda(), qr.cuda(), lat.cuda(), bt, cl, scale)
    assert torch.equal(got, again)


def test_mla_decode_bf16_fewer_than_16_heads():
    ops = _ops()
    H, r, dr, bs = 5, 512, 64, 16
    lens = [130, 700, 31]
    case = deal_blocks(lens, bs, np.random.default_rng(9), pad_blocks=1)
    qa = (_randn((3, H, r), 70, torch.float32) * 0.2).to(torch.bfloat16)
    qr = _randn((3, H, dr), 71, torch.bfloat16)
    lat = _randn((case.num_blocks, bs, r + dr), 72, torch.bfloat16)
    want = _oracle().mla_decode(qa, qr, lat, case.block_tables, case.context_lens, 0.07)
    got = ops.mla_decode(qa.cuda(), qr.cuda(), lat.cuda(), torch.from_numpy(case.block_tables).cuda(),
                         torch.from_numpy(case.context_lens).cuda(), 0.07)
    ops.check_status()
    assert_close(got, want, torch.bfloat16)


# ----------------------------------------------------------------------------- fused glue kernels
@pytest.mark.parametrize("dim", [512, 2048, 1000])      # bf16: 512 and 2048 take the warp-per-row kernel
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_add_rmsnorm_matches_oracle(dtype, dim):
    ops, orc = _ops(), _oracle()
    x, res = _randn((37, dim), 1, dtype), _randn((37, dim), 2, torch.float32)
    w = _randn((dim,), 3, torch.float32)
    want = orc.rms_norm(x, w, 1e-5)
    got = ops.add_rmsnorm(x.cuda(), w.cuda(), 1e-5)
    tol = 1e-5 if dtype == torch.float32 else 2e-2
    assert (got.float().cpu() - want.float()).abs().max().item() <= tol
    for r in (res, res.to(dtype)):     # residual in fp32 (first layer) or in the activation dtype
        wy, wr = orc.rms_norm(x, w, 1e-5, r)
        gy, gr = ops.add_rmsnorm(x.cuda(), w.cuda(), 1e-5, r.cuda())
        assert gy.dtype == dtype and gr.dtype == dtype
        assert (gy.float().cpu() - wy.float()).abs().max().item() <= tol
        assert (gr.float().cpu() - wr.float()).abs().max().item() <= (1e-6 if dtype == torch.float32 else 2e-2)


@pytest.mark.parametrize("Hq,Hkv,D", [(8, 2, 64), (8, 4, 64), (4, 2, 128), (16, 8, 32), (2, 1, 256)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_qk_norm_rope_store_matches_oracle_and_scatter(dtype, Hq, Hkv, D):
    """Against the oracle's RMSNorm-over-the-whole-vector + RoPE (model/attention/GQA.py:81-94) and its
    store_kvcache, including a padded (-1) slot.  Widths that are multiples of 256 take the
    warp-per-token bf16 kernel, (8, 2, 64) and fp32 the general one."""
    ops, orc = _ops(), _oracle()
    T, bs, nb = 29, 16, 4
    qkv = _randn((T, (Hq + 2 * Hkv) * D), 5, dtype)
    qw, kw = _randn((Hq * D,), 6, torch.float32), _randn((Hkv * D,), 7, torch.float32)
    table = orc.rope_table(10000.0, D, 128)
    pos = torch.from_numpy(np.random.default_rng(0).integers(0, 128, size=T).astype(np.int64))
    slots = torch.from_numpy(np.random.default_rng(1).permutation(nb * bs)[:T].astype(np.int64))
    slots[3] = -1

    def vec_norm(x, w):     # the reference's nn.RMSNorm(eps=None) with an fp32 weight
        return torch.nn.functional.rms_norm(x, (x.shape[-1],), w, None).to(dtype)
    q = vec_norm(qkv[:, :Hq * D], qw).view(T, Hq, D).transpose(0, 1)
    k = vec_norm(qkv[:, Hq * D:(Hq + Hkv) * D], kw).view(T, Hkv, D).transpose(0, 1)
    v = qkv[:, (Hq + Hkv) * D:].view(T, Hkv, D)
    want_q = orc.apply_rope(q.float(), pos, table).transpose(0, 1).to(dtype)
    want_k = orc.apply_rope(k.float(), pos, table).transpose(0, 1).to(dtype)
    kc_ref, vc_ref = torch.zeros(nb, bs, Hkv, D, dtype=dtype), torch.zeros(nb, bs, Hkv, D, dtype=dtype)
    orc.store_kvcache(want_k, v, kc_ref, vc_ref, slots)
    kc, vc = torch.zeros_like(kc_ref).cuda(), torch.zeros_like(vc_ref).cuda()
    gq, gk, gv = ops.qk_norm_rope_store(qkv.cuda(), qw.cuda(), kw.cuda(), table.cuda(), pos.cuda(), Hq, Hkv, D,
                                        kc, vc, slots.cuda())
    ops.check_status()
    tol = 2e-5 if dtype == torch.float32 else 4e-2     # bf16: one rounding step of values up to ~4
    assert (gq.float().cpu() - want_q.float()).abs().max().item() <= tol
    assert (gk.float().cpu() - want_k.float()).abs().max().item() <= tol
    assert torch.equal(gv.cpu(), v)
    assert torch.equal(vc.cpu(), vc_ref)
    assert torch.equal(kc.view(-1, Hkv, D)[slots[slots >= 0].cuda()].cpu(), gk.cpu()[slots >= 0])
    assert (kc.view(-1, Hkv, D).float().abs().sum(dim=(1, 2)) > 0).sum().item() == T - 1


@pytest.mark.parametrize("H,hd,dr,r,width", [(16, 128, 64, 512, 128), (4, 64, 32, 128, 64), (3, 64, 64, 72, 64),
                                             (16, 128, 64, 512, 64)])
def test_mla_prologue_matches_oracle(H, hd, dr, r, width):
    """q = [q_nope | RoPE(q_rope)] and the latent row [kv_norm(c) | RoPE(k_rope)] against the oracle's
    RMSNorm and RoPE (model/attention/MLA.py:114-131), with the rope table sliced to rope_dim columns as
    the reference slices it (a table wider than rope_dim yields cosines in the "sin" half), and the
    scatter into the latent cache including a padded (-1) slot."""
    ops, orc = _ops(), _oracle()
    dtype = torch.bfloat16
    T, bs, nb = 37, 16, 4
    qf = _randn((T, H * (hd + dr)), 11, dtype)
    kvp = _randn((T, r + dr), 12, dtype)
    w = _randn((r,), 13, torch.float32)
    table = orc.rope_table(10000.0, width, 96)
    pos = torch.from_numpy(np.random.default_rng(2).integers(0, 96, size=T).astype(np.int64))
    slots = torch.from_numpy(np.random.default_rng(3).permutation(nb * bs)[:T].astype(np.int64))
    slots[5] = -1
    q_nope = qf[:, :H * hd].view(T, H, hd)
    q_rope = orc.apply_rope(qf[:, H * hd:].view(T, H, dr).transpose(0, 1).float(), pos, table).transpose(0, 1)
    want_q = torch.cat([q_nope, q_rope.to(dtype)], dim=-1)
    c = torch.nn.functional.rms_norm(kvp[:, :r], (r,), w, None).to(dtype)   # nn.RMSNorm(eps=None), fp32 weight
    pe = orc.apply_rope(kvp[:, r:].float().unsqueeze(0), pos, table).squeeze(0).to(dtype)
    want_rows = torch.cat([c, pe], dim=-1)

    cache = torch.zeros(nb, bs, r + dr, dtype=dtype).cuda()
    gq, grows = ops.mla_prologue(qf.cuda(), kvp.cuda(), w.cuda(), table.cuda(), pos.cuda(), H, hd, dr, r,
                                 cache, slots.cuda())
    ops.check_status()
    assert torch.equal(gq[..., :hd].cpu(), q_nope)
    tol = 4e-2                                            # one bf16 rounding step of values up to ~4
    assert (gq.float().cpu() - want_q.float()).abs().max().item() <= tol
    assert (grows.float().cpu() - want_rows.float()).abs().max().item() <= tol
    # nearly every element rounds the same way as the tensor-op form
    assert (gq.cpu() == want_q).float().mean().item() > 0.99
    assert (grows.cpu() == want_rows).float().mean().item() > 0.99
    flat = cache.view(-1, r + dr)
    assert torch.equal(flat[slots[slots >= 0].cuda()].cpu(), grows.cpu()[slots >= 0])
    assert (flat.float().abs().sum(dim=1) > 0).sum().item() == T - 1
    # without a cache nothing is scattered and the rows are the same
    gq2, grows2 = ops.mla_prologue(qf.cuda(), kvp.cuda(), w.cuda(), table.cuda(), pos.cuda(), H, hd, dr, r)
    assert torch.equal(gq2, gq) and torch.equal(grows2, grows)


def test_mla_prologue_rejects_bad_arguments():
    ops = _ops()
    dtype = torch.bfloat16
    qf, kvp = torch.zeros(4, 4 * 96, dtype=dtype).cuda(), torch.zeros(4, 160, dtype=dtype).cuda()
    w, table = torch.ones(128).cuda(), torch.zeros(8, 64).cuda()
    pos = torch.zeros(4, dtype=torch.int64).cuda()
    with pytest.raises(ValueError):
        ops.mla_prologue(qf.float(), kvp.float(), w, table, pos, 4, 64, 32, 128)
    with pytest.raises(ValueError):
        ops.mla_prologue(qf, kvp[:, :100], w, table, pos, 4, 64, 32, 128)
    with pytest.raises(RuntimeError):                      # rope_dim 24: 3 chunks, not a power of two
        ops.mla_prologue(torch.zeros(4, 4 * 88, dtype=dtype).cuda(), torch.zeros(4, 152, dtype=dtype).cuda(), w,
                         table, pos, 4, 64, 24, 128)
    # a position outside the table is clamped and reported
    pos[2] = 99
    ops.mla_prologue(qf, kvp, w, table, pos, 4, 64, 32, 128)
    with pytest.raises(RuntimeError):
        ops.check_status()


@pytest.mark.parametrize("with_plan", [False, True])
def test_prefill_shared_tail_equals_expanded_keys(with_plan):
    """Keys in two parts (per-head columns + a rotary tail shared by all heads, MLA.py:131) give the
    same output, bit for bit, as the same kernel run on keys with the tail copied into every head;
    the parts are strided views of wider buffers, as the model passes them."""
    ops = _ops()
    H, hd, dr = 4, 128, 64
    lens_q, lens_k = [70, 1, 200, 33], [70, 1, 260, 33]
    cu_q = torch.tensor(np.concatenate([[0], np.cumsum(lens_q)]).astype(np.int32)).cuda()
    cu_k = torch.tensor(np.concatenate([[0], np.cumsum(lens_k)]).astype(np.int32)).cuda()
    Tq, Tk = sum(lens_q), sum(lens_k)
    q = _randn((Tq, H, hd + dr), 21, torch.bfloat16).cuda()
    kv = _randn((Tk, 2 * H * hd), 22, torch.bfloat16).cuda()
    rows = _randn((Tk, 512 + dr), 23, torch.bfloat16).cuda()
    k_head, v = kv[:, :H * hd].view(Tk, H, hd), kv[:, H * hd:].view(Tk, H, hd)
    tail = rows[:, 512:]
    k_full = torch.cat([k_head, tail.unsqueeze(1).expand(-1, H, dr)], dim=-1)
    plan = None
    if with_plan:
        rows_per_tile = ops.prefill_tile_rows(H, H, hd + dr, hd, torch.bfloat16)
        plan = ops.prefill_plan(cu_q, Tq, max(lens_q), rows_per_tile)
    want = ops.prefill_varlen(q, k_full, v.contiguous(), cu_q, cu_k, max(lens_q), max(lens_k), 192 ** -0.5, plan=plan)
    got = ops.prefill_varlen_shared_tail(q, k_head, tail, v, cu_q, cu_k, max(lens_q), 192 ** -0.5, plan=plan)
    ops.check_status()
    assert torch.equal(got, want)
    assert got.float().abs().sum().item() > 0


def _moe_rows(T, K, E, seed):
    """A consistent grouping: every token picks K distinct experts; rows sorted by (expert, token)."""
    rng = np.random.default_rng(seed)
    sel = np.stack([np.sort(rng.choice(E, size=K, replace=False)) for _ in range(T)])        # [T, K]
    flat_e, flat_t = sel.reshape(-1), np.repeat(np.arange(T), K)
    order = np.lexsort((flat_t, flat_e))
    inv = np.empty(T * K, dtype=np.int32)
    inv[order] = np.arange(T * K, dtype=np.int32)
    return (torch.from_numpy(flat_e[order].astype(np.int32)).cuda(), torch.from_numpy(inv.reshape(T, K)).cuda())


@pytest.mark.parametrize("dtype,F", [(torch.bfloat16, 704), (torch.bfloat16, 100), (torch.float32, 96)])
def test_swiglu_matches_the_tensor_op_sequence(dtype, F):
    """silu(h1 + b1) * (h3 + b3) of mlp.py:61-67 with the roundings of add -> silu -> mul on tensors."""
    import torch.nn.functional as Fn
    ops = _ops()
    rows, E = 333, 5
    h = _randn((rows, 2 * F), 11, dtype).cuda()
    bias = _randn((E, 2 * F), 12, dtype).cuda()
    experts = torch.from_numpy(np.sort(np.random.default_rng(3).integers(0, E, size=rows)).astype(np.int32)).cuda()
    for b, e in ((None, None), (bias, experts), (bias[:1].contiguous(), None)):
        hb = h if b is None else h + (b[e.long()] if e is not None else b[0])
        want = Fn.silu(hb[:, :F]) * hb[:, F:]
        got = ops.swiglu(h, b, e)
        assert got.shape == want.shape and got.dtype == dtype
        err = (got.float() - want.float()).abs()
        assert (err <= 1e-2 * want.float().abs() + 1e-5).all(), err.max().item()   # at most one rounding step


@pytest.mark.parametrize("dtype,d", [(torch.bfloat16, 1024), (torch.bfloat16, 100), (torch.float32, 64)])
def test_moe_combine_adds_in_ascending_expert_order(dtype, d):
    """Bit-equal to: (y + b2[expert]) * w, regrouped per token, summed left to right in the dtype, + shared
    (the accumulation order of moe.py:312-339 and 272-273)."""
    ops = _ops()
    T, K, E = 77, 3, 6
    experts, inv = _moe_rows(T, K, E, 4)
    y = _randn((T * K, d), 21, dtype).cuda()
    b2 = _randn((E, d), 22, dtype).cuda()
    w = torch.rand(T * K, generator=torch.Generator().manual_seed(23)).to(dtype).cuda()
    shared = _randn((T, d), 24, dtype).cuda()
    for bias, sh in ((b2, shared), (None, None), (b2, None)):
        rows = y if bias is None else y + bias[experts.long()]
        yt = (rows * w.unsqueeze(1))[inv.long().reshape(-1)].view(T, K, d)
        want = yt[:, 0]
        for k in range(1, K):
            want = want + yt[:, k]
        if sh is not None:
            want = want + sh
        got = ops.moe_combine(y, bias, experts, w, inv, sh)
        if dtype == torch.bfloat16:
            assert torch.equal(got, want)
        else:
            assert (got - want).abs().max().item() <= 1e-5


def test_moe_route_many_ctas_is_a_stable_counting_sort():
    """5,000 tokens (20 CTAs), 16 experts top-2, and 64 experts top-8: rows ordered by (expert, token),
    offsets = cumulative counts, slot_to_row inverts the order; selection equals a host top-k."""
    ops = _ops()
    for T, E, K in ((5000, 16, 2), (1000, 64, 8), (256, 16, 2), (257, 3, 3)):
        g = torch.Generator().manual_seed(T + E)
        logits = torch.randn(T, E, generator=g).cuda()             # fp32: no ties
        bias = (0.1 * torch.randn(E, generator=g)).cuda()
        tok, experts, w, offs, inv = ops.moe_route(logits, bias, K)
        ops.check_status()
        assert torch.equal(offs, experts.bincount(minlength=E).cumsum(0).int())
        key = experts.long() * T + tok.long()
        assert (key[1:] > key[:-1]).all()
        want_sel = torch.topk(logits + bias, K, dim=-1).indices.sort(dim=1).values
        rows = inv.long().reshape(-1)
        assert torch.equal(experts[rows].view(T, K).long(), want_sel)
        assert torch.equal(tok[rows].view(T, K).long(), torch.arange(T, device="cuda").view(T, 1).expand(T, K))
        scores = torch.sigmoid(logits).gather(1, want_sel)
        want_w = scores / (scores.sum(-1, keepdim=True) + 1e-10) if K > 1 else scores
        assert (w[rows].view(T, K) - want_w).abs().max().item() <= 1e-6


def _grouped_reference(x, w, offs, bias, swiglu):
    """The CPU oracle's per-expert loop (fp32 products on the host, bf16 roundings of the tensor-op sequence)."""
    from oracle.moe import grouped_linear
    return grouped_linear(x, w, offs.cpu().tolist(), bias, swiglu).to(x.device)


@pytest.mark.parametrize("counts,k,n,swiglu", [
    ([12, 0, 31, 7, 16, 1, 64, 25], 1024, 704, True),        # decode-like: one pass per expert
    ([12, 0, 31, 7, 16, 1, 64, 25], 704, 1024, False),
    ([150, 3, 0, 0, 70, 9], 256, 200, True),                 # > 64 rows in the small configuration: several passes
    ([150, 3, 0, 0, 70, 9], 200, 1000, False),               # ragged K (200 = 3 slabs + 8) and ragged n_out
    ([700, 90, 300, 10], 512, 192, True),                    # large batch: 256 rows per pass, several passes
    ([700, 90, 300, 10], 192, 520, False),
    ([0, 0, 5], 64, 64, False),
    ([915, 1, 0, 1300, 128, 129, 127, 400], 1024, 704, True),    # compute-bound kernel: ragged row tiles, 5.5 column tiles
    ([915, 1, 0, 1300, 128, 129, 127, 400], 704, 1024, False),
])
def test_moe_grouped_gemm_matches_per_expert_matmuls(counts, k, n, swiglu):
    ops = _ops()
    E, R = len(counts), sum(counts)
    offs = torch.tensor(np.cumsum(counts), dtype=torch.int32, device="cuda")
    x = _randn((R, k), 31, torch.bfloat16).cuda()
    w = (_randn((E, 2 * n if swiglu else n, k), 32, torch.float32) * k ** -0.5).bfloat16().cuda()
    bias = _randn((E, 2 * n if swiglu else n), 33, torch.bfloat16).cuda()
    for b in (bias, None):
        got = ops.moe_grouped_gemm(x, w, offs, b, swiglu=swiglu)
        ops.check_status()
        want = _grouped_reference(x, w, offs, b, swiglu)
        assert got.shape == want.shape
        err = (got.float() - want.float()).abs()
        assert (err <= 2e-2 * want.float().abs() + 2e-2).all(), err.max().item()
    again = ops.moe_grouped_gemm(x, w, offs, bias, swiglu=swiglu)
    assert torch.equal(again, ops.moe_grouped_gemm(x, w, offs, bias, swiglu=swiglu))


@pytest.mark.parametrize("counts,k,n", [([256, 257, 384, 385, 128, 1, 0, 640], 128, 264),                          # weights stay in L2: short tiles last
                                        ([300, 1, 257, 0, 700, 128, 129, 256, 90, 385, 511, 40, 65], 2048, 1024)])   # 109 MB of them: in order
def test_moe_grouped_gemm_row_tiles_of_one_and_two_halves(counts, k, n):
    ops = _ops()
    offs = torch.tensor(np.cumsum(counts), dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn(sum(counts), k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(len(counts), 2 * n, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    got, want = ops.moe_grouped_gemm(x, w, offs, None, swiglu=True), _grouped_reference(x, w, offs, None, True)
    ops.check_status()
    assert ((got.float() - want.float()).abs() <= 2e-2 * want.float().abs() + 2e-2).all()


@pytest.mark.parametrize("swiglu,big", [(True, False), (False, False), (True, True), (False, True)])
def test_moe_grouped_gemm_dense_tail_is_one_more_weight_set(swiglu, big):
    """Rows after the grouped ones that all use weight set E (a shared expert in the same launch), in
    chunks of 64; 150 tail rows = two full chunks and a ragged one.  ``big``: many rows per expert, served by
    the compute-bound kernel, where the tail is one more group of row tiles."""
    ops = _ops()
    counts, tail, k, n = [12, 0, 31, 7, 16, 1, 60, 25], 150, 256, 192
    if big:
        counts, tail = [300, 0, 131, 700, 16, 1, 260, 425], 917
    E, R = len(counts), sum(counts)
    offs = torch.tensor(np.cumsum(counts), dtype=torch.int32, device="cuda")
    x = _randn((R + tail, k), 41, torch.bfloat16).cuda()
    w = (_randn((E + 1, 2 * n if swiglu else n, k), 42, torch.float32) * k ** -0.5).bfloat16().cuda()
    bias = _randn((E + 1, 2 * n if swiglu else n), 43, torch.bfloat16).cuda()
    got = ops.moe_grouped_gemm(x, w, offs, bias, swiglu=swiglu, dense_rows=tail)
    ops.check_status()
    all_offs = torch.cat([offs, torch.tensor([R + tail], dtype=torch.int32, device="cuda")])
    want = _grouped_reference(x, w, all_offs, bias, swiglu)
    err = (got.float() - want.float()).abs()
    assert (err <= 2e-2 * want.float().abs() + 2e-2).all(), err.max().item()
    # routing with the identity tail: the gather index of the tail rows
    logits = _randn((100, 8), 44, torch.bfloat16).cuda()
    tok, experts, wts, o2, inv = ops.moe_route(logits, torch.zeros(8, device="cuda"), 2, identity_tail=True)
    assert tok.numel() == 300 and torch.equal(tok[200:], torch.arange(100, device="cuda", dtype=torch.int32))
    tok2 = ops.moe_route(logits, torch.zeros(8, device="cuda"), 2)[0]
    assert torch.equal(tok[:200], tok2)


# ----------------------------------------------------------------------------- empty inputs
def test_empty_inputs_are_no_ops():
    """Zero tokens / zero sequences through every entry point: success, nothing launched or written."""
    from llm_from_scratch_b200._lib import lib, DTYPE_BF16
    ops = _ops()
    dev = torch.device("cuda")
    kc = torch.ones(2, 16, 2, 64, dtype=torch.bfloat16, device=dev)
    vc = torch.ones_like(kc)
    empty_kv = torch.empty(0, 2, 64, dtype=torch.bfloat16, device=dev)
    ops.store_kvcache(empty_kv, empty_kv, kc, vc, torch.empty(0, dtype=torch.int64, device=dev))
    assert (kc == 1).all() and (vc == 1).all()
    s = torch.cuda.current_stream().cuda_stream
    assert lib.b200_paged_decode_gqa(None, None, None, None, None, 1, None, 0, 8, 2, 64, 16, 2, 0.125, None, 0,
                                     DTYPE_BF16, None, s) == 0
    assert lib.b200_mla_decode(None, None, None, None, None, 1, None, 0, 16, 512, 64, 16, 2, 0.07, None, 0,
                               DTYPE_BF16, None, s) == 0
    assert lib.b200_prefill_varlen(None, None, None, None, 0, 0, 0, 0, 0, None, None, 0, 0, 0, 8, 2, 64, 64, 0.125,
                                   None, None, None, 0, 0, 0, None, None, 0, 0, DTYPE_BF16, None, s) == 0
    # a batch whose contexts are all empty: zero rows, no block is read
    q = torch.randn(3, 8, 64, device=dev).bfloat16()
    bt = torch.full((3, 4), -1, dtype=torch.int32, device=dev)
    out = ops.paged_decode_gqa(q, kc, vc, bt, torch.zeros(3, dtype=torch.int64, device=dev), 0.125)
    ops.check_status()
    assert (out == 0).all()


# ----------------------------------------------------------------------------- sampler
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sample_greedy_is_argmax_with_first_maximum(dtype):
    ops = _ops()
    logits = _randn((37, 1000), 91, dtype).cuda()
    logits[3, 10] = logits[3, 700] = 50.0            # a tie: the lower index wins
    logits[5] = 0.0                                   # a whole row of equal values
    got = ops.sample(logits, None, seed=1, offset=1)
    assert torch.equal(got, logits.float().argmax(dim=-1)) and got[3].item() == 10 and got[5].item() == 0
    temps = torch.zeros(37, device="cuda")
    assert torch.equal(ops.sample(logits, temps, seed=1, offset=2), got)      # T = 0 rows are greedy too
    wide = torch.full((4, 1500), -1.0, dtype=dtype, device="cuda")            # rows with a stride
    view = wide[:, :1000]
    view[:, 123] = 2.0
    assert ops.sample(view, None, 0, 0).tolist() == [123] * 4


def test_sample_with_temperature_follows_the_softmax_distribution():
    """20,000 rows with the same 8 logits: the draw frequencies match softmax(logits / T) within four
    standard deviations (the reference's exponential race, utils/sampler.py:48-51, has that law); the
    stream is a function of (seed, offset) only."""
    ops = _ops()
    n, T = 20000, 0.7
    base = torch.tensor([2.0, 1.0, 0.5, 0.0, -0.5, -1.0, 3.0, -4.0])
    logits = base.repeat(n, 1).cuda()
    temps = torch.full((n,), T, device="cuda")
    got = ops.sample(logits, temps, seed=123, offset=7)
    freq = torch.bincount(got.cpu(), minlength=8).double() / n
    p = torch.softmax(base.double() / T, dim=0)
    sigma = (p * (1 - p) / n).sqrt()
    assert ((freq - p).abs() <= 4 * sigma + 1e-4).all(), (freq, p)
    assert torch.equal(got, ops.sample(logits, temps, seed=123, offset=7))
    assert not torch.equal(got, ops.sample(logits, temps, seed=123, offset=8))
    mixed = temps.clone()
    mixed[::2] = 0.0                                                          # greedy and sampled rows together
    out = ops.sample(logits, mixed, seed=5, offset=1)
    assert (out[::2] == 6).all() and (out[1::2] != 6).any()


def test_decode_advance_steps_the_decode_metadata():
    """input id = sampled token, context length + 1 and the slot of the new position from the block table,
    exactly what prepare_decode computes on the host for the next step (model_runner.py:253-278); a table
    that does not list the needed block gives slot -1 and a reported bounds error; rows past n untouched."""
    ops = _ops()
    bs, nb, n = 16, 64, 5
    lens = torch.tensor([1, 15, 16, 17, 47, 99, 99], dtype=torch.int64)
    tables = torch.from_numpy(np.random.default_rng(5).permutation(nb)[:7 * 4].reshape(7, 4).astype(np.int32))
    sampled = torch.tensor([11, 12, 13, 14, 15, 16, 17], dtype=torch.int64)
    ids, slots = torch.full((7,), -5, dtype=torch.int64), torch.full((7,), -5, dtype=torch.int64)
    hist = torch.full((7,), -5, dtype=torch.int64)
    d = [t.cuda() for t in (sampled, ids, lens.clone(), slots, tables, hist)]
    ops.decode_advance(d[0][:n], d[1], d[2], d[3], d[4], bs, nb, d[5])
    ops.check_status()
    new_len = lens[:n] + 1
    want_slots = tables[torch.arange(n), (new_len - 1) // bs].long() * bs + (new_len - 1) % bs
    assert d[1].cpu().tolist() == [11, 12, 13, 14, 15, -5, -5]
    assert d[2].cpu().tolist() == new_len.tolist() + [99, 99]
    assert d[3].cpu().tolist() == want_slots.tolist() + [-5, -5]
    assert d[5].cpu().tolist() == [11, 12, 13, 14, 15, -5, -5]
    # length 64 -> 65 needs block 4 of a 4-entry table: slot -1, error reported (and cleared by the read)
    lens2 = torch.tensor([64], dtype=torch.int64).cuda()
    ops.decode_advance(d[0][:1], d[1], lens2, d[3], d[4], bs, nb)
    assert d[3][0].item() == -1
    with pytest.raises(RuntimeError):
        ops.check_status()


def test_mla_decode_benchmark_shape_sampled_rows():
    """The MLA benchmark's decode batch at full size (240 sequences, contexts uniform [512,16384], latent
    512 + 64, 2.07 M context tokens): a sample of rows against the oracle, and a second call gives the
    same bits (fixed cut, no atomics)."""
    from llm_from_scratch_b200.workloads import c4_decode_case
    ops = _ops()
    case = c4_decode_case()
    H, r, dr, bs = 16, 512, 64, 16
    g = torch.Generator(device="cuda").manual_seed(4)
    lat = (torch.randn(case.num_blocks, bs, r + dr, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    qa = (torch.randn(case.batch, H, r, generator=g, device="cuda") * 0.2).to(torch.bfloat16)
    qr = torch.randn(case.batch, H, dr, generator=g, device="cuda", dtype=torch.bfloat16)
    bt, cl = torch.from_numpy(case.block_tables).cuda(), torch.from_numpy(case.context_lens).cuda()
    scale = 192 ** -0.5
    out = ops.mla_decode(qa, qr, lat, bt, cl, scale)
    ops.check_status()
    assert torch.isfinite(out.float()).all()
    assert torch.equal(out, ops.mla_decode(qa, qr, lat, bt, cl, scale))
    for b in [0, 7, 123, 239, int(np.argmax(case.context_lens)), int(np.argmin(case.context_lens))]:
        L = int(case.context_lens[b])
        nblk = (L + bs - 1) // bs
        ids = torch.from_numpy(case.block_tables[b, :nblk].astype(np.int64)).cuda()
        want = _oracle().mla_decode(qa[b:b + 1].cpu(), qr[b:b + 1].cpu(), lat[ids].cpu(), [list(range(nblk))], [L], scale)
        assert_close(out[b:b + 1], want, torch.bfloat16)


def test_mla_prefill_benchmark_step_sampled_sequences():
    """The MLA benchmark's prefill batch at full size (16 prompts, lengths uniform [256,4096], 16 heads,
    192/128 head dims, keys = per-head columns + the rotary tail shared by all heads, both strided views):
    the shortest, the longest and one more sequence against the oracle on expanded keys."""
    ops = _ops()
    rng = np.random.default_rng(4)
    lens = rng.integers(256, 4097, size=16)
    T, H, hd, dr, r = int(lens.sum()), 16, 128, 64, 512
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn(T, H, hd + dr, generator=g, device="cuda", dtype=torch.bfloat16)
    kv = torch.randn(T, 2 * H * hd, generator=g, device="cuda", dtype=torch.bfloat16)
    rows = torch.randn(T, r + dr, generator=g, device="cuda", dtype=torch.bfloat16)
    k_head, v, tail = kv[:, :H * hd].view(T, H, hd), kv[:, H * hd:].view(T, H, hd), rows[:, r:]
    cu_np = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cu = torch.from_numpy(cu_np).cuda()
    mx = int(lens.max())
    plan = ops.prefill_plan(cu, T, mx, ops.prefill_tile_rows(H, H, hd + dr, hd, torch.bfloat16))
    scale = (hd + dr) ** -0.5
    out = ops.prefill_varlen_shared_tail(q, k_head, tail, v, cu, cu, mx, scale, plan=plan)
    ops.check_status()
    assert torch.isfinite(out.float()).all()
    for s in sorted({int(np.argmin(lens)), int(np.argmax(lens)), 5}):
        a, b = int(cu_np[s]), int(cu_np[s + 1])
        k_full = torch.cat([k_head[a:b], tail[a:b].unsqueeze(1).expand(-1, H, dr)], dim=-1).cpu()
        one = torch.tensor([0, b - a], dtype=torch.int32)
        want = _oracle().prefill_varlen(q[a:b].cpu(), k_full, v[a:b].cpu(), one, one, scale)
        assert_close(out[a:b], want, torch.bfloat16)


# ----------------------------------------------------------------------------- bounded waits
def test_a_barrier_wait_that_runs_out_is_reported_and_leaves_the_device_usable():
    """The give-up path shared by the tcgen05 / TMA kernels, run on purpose by the diagnostic entry point: a wait
    with a short poll limit times out, the CTA's other waiter leaves through the abort flag, tensor memory is
    freed, the status word reads B200_ERR_TIMEOUT — and the kernels that allocate all 512 tensor-memory
    columns of an SM run correctly right afterwards on every SM."""
    from oracle import attention as orc
    ops = _ops()
    ops.check_status()
    for limit in (64, 1000):
        res = ops.selftest_bounded_wait(limit)
        assert res[0] == 0 and res[1] == limit, res          # ran out exactly at its limit
        assert res[2] == 0 and 0 < res[3] < (1 << 22), res   # left early, through the flag
        assert res[4] == 1, res
        assert ops.read_status_code() == -9                  # B200_ERR_TIMEOUT, and the word is cleared
        assert ops.read_status_code() == 0
    # a tcgen05 prefill on every SM (300 CTAs of 512 tensor-memory columns each) still runs and is right
    Hq, Hkv, D = 8, 2, 128
    lens = [700, 1, 333, 2048, 129]
    T = sum(lens)
    q, k, v = (_randn((T, h, D), 50 + i, torch.bfloat16) for i, h in enumerate((Hq, Hkv, Hkv)))
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32)
    got = ops.prefill_varlen(q.cuda(), k.cuda(), v.cuda(), cu.cuda(), cu.cuda(), max(lens), max(lens), D ** -0.5)
    ops.check_status()
    rows = torch.tensor([0, 699, 700, 701, 1033, 1034, 2000, T - 130, T - 1])
    want = orc.prefill_varlen(q, k, v, cu, cu, D ** -0.5)
    assert (got.float().cpu()[rows] - want[rows]).abs().max().item() <= 2e-2


# ----------------------------------------------------------------------------- split contexts merged in the launch
def test_split_contexts_are_merged_inside_the_decode_launch_and_counters_return_to_zero():
    """Contexts cut across thread blocks are merged by the last piece to arrive: calls of different shapes share
    one scratch buffer back to back, every call matches the oracle, repeated calls are bit-identical (the merge
    order is fixed), and the arrival counters at the head of the buffer are zero after every call.  A batch with
    more (sequence, KV head) pairs than counters takes the separate merge kernel and matches as well."""
    ops, orc = _ops(), _oracle()
    from llm_from_scratch_b200.workloads import deal_blocks
    shapes = [((32, 8, 128), [9000, 3, 4100, 0, 16, 17, 2500]), ((16, 4, 64), [700, 1300, 250, 1, 999, 64] * 8),
              ((8, 8, 32), [5000, 5000, 33]), ((32, 8, 128), [6000, 1])]
    for (Hq, Hkv, D), lens in shapes:
        case = deal_blocks(lens, 16, np.random.default_rng(len(lens)), pad_blocks=2)
        q = _randn((len(lens), Hq, D), 61, torch.bfloat16)
        kc = _randn((case.num_blocks, 16, Hkv, D), 62, torch.bfloat16)
        vc = _randn((case.num_blocks, 16, Hkv, D), 63, torch.bfloat16)
        bt, cl = torch.from_numpy(case.block_tables).cuda(), torch.from_numpy(case.context_lens).cuda()
        got = ops.paged_decode_gqa(q.cuda(), kc.cuda(), vc.cuda(), bt, cl, D ** -0.5)
        again = ops.paged_decode_gqa(q.cuda(), kc.cuda(), vc.cuda(), bt, cl, D ** -0.5)
        ops.check_status()
        want = orc.paged_decode_gqa(q, kc, vc, case.block_tables, case.context_lens, D ** -0.5)
        assert (got.float().cpu() - want).abs().max().item() <= 2e-2
        assert torch.equal(got, again)
        ws = ops._workspaces[(torch.cuda.current_device(), "decode")]
        assert int(ws[:256 * 1024].view(torch.int32).abs().sum().item()) == 0
    # 9,000 sequences x 8 KV heads: more pairs than the 65,536 counters
    lens = [40] * 8990 + [3000] * 10
    case = deal_blocks(lens, 16, np.random.default_rng(5), pad_blocks=2)
    q = _randn((len(lens), 8, 64), 64, torch.bfloat16)
    kc = _randn((case.num_blocks, 16, 8, 64), 65, torch.bfloat16)
    bt, cl = torch.from_numpy(case.block_tables).cuda(), torch.from_numpy(case.context_lens).cuda()
    got = ops.paged_decode_gqa(q.cuda(), kc.cuda(), kc.cuda(), bt, cl, 0.125)
    ops.check_status()
    rows = [0, 4000, 8989, 8990, 8999]
    want = orc.paged_decode_gqa(q[rows], kc, kc, case.block_tables[rows], case.context_lens[rows], 0.125)
    assert (got.float().cpu()[rows] - want).abs().max().item() <= 2e-2


# ----------------------------------------------------------------------------- greedy head
@pytest.mark.parametrize("rows,vocab,d", [(1, 32000, 1024), (7, 1000, 256), (64, 32000, 1024), (65, 5000, 512),
                                          (256, 32000, 1024), (300, 777, 128)])
def test_lm_head_argmax_equals_argmax_of_the_bf16_logits(rows, vocab, d):
    """Fused head (projection + first-maximum argmax, logits never written) against the CPU: logits in fp32 from
    the bf16 operands, + bias, rounded to bf16 once (what the reference's biased bf16 Linear returns), argmax.
    Rows whose two largest bf16 logits are closer than two rounding steps may legitimately pick either (the
    accumulation order differs); there the chosen logit must still be within that distance of the maximum."""
    ops = _ops()
    h = (_randn((rows, d), 71, torch.float32)).bfloat16()
    w = (_randn((vocab, d), 72, torch.float32) * d ** -0.5).bfloat16()
    b = (_randn((vocab,), 73, torch.float32) * 0.1).bfloat16()
    for bias in (b, None):
        got = ops.lm_head_argmax(h.cuda(), w.cuda(), None if bias is None else bias.cuda()).cpu()
        ops.check_status()
        logits = h.float() @ w.float().t()
        if bias is not None:
            logits = logits + bias.float()
        logits = logits.bfloat16().float()
        want = logits.argmax(dim=-1)
        top = logits.max(dim=-1).values
        chosen = logits.gather(1, got.view(-1, 1)).squeeze(1)
        step = top.abs() * 2.0 ** -7
        assert (got >= 0).all() and (got < vocab).all()
        assert ((top - chosen) <= 2 * step).all(), (top - chosen).max().item()
        assert (got == want).float().mean().item() >= 0.97
    # equal maxima: the lowest index wins
    w2 = w.clone()
    w2[5] = w2[900 % vocab] = w2[3]
    got = ops.lm_head_argmax(h.cuda(), w2.cuda(), None).cpu()
    logits = (h.float() @ w2.float().t()).bfloat16().float()
    tie_rows = logits.argmax(dim=-1) == 3
    assert (got[tie_rows] == 3).all()


# ----------------------------------------------------------------------------- gate projection + routing in one launch
@pytest.mark.parametrize("T,E,K,d,tail,gather", [(1, 16, 2, 1024, True, True), (7, 16, 2, 1024, True, True),
                                                  (32, 16, 2, 1024, False, True), (200, 16, 2, 1024, True, False),
                                                  (256, 32, 4, 2048, True, False), (33, 64, 8, 512, False, True),
                                                  (9, 4, 2, 128, True, True)])
def test_gate_projection_and_routing_in_one_launch(T, E, K, d, tail, gather):
    """b200_moe_gate_route against the two-step form (bf16 gate logits computed on the CPU in fp32 and rounded
    once, then b200_moe_route): the sort invariants always hold; selection and weights agree wherever the two
    logit computations do not disagree about a near-tie; the gathered rows are x[sorted_token]; two calls in a
    row share the scratch (its ticket returns to zero)."""
    ops = _ops()
    x = _randn((T, d), 81, torch.bfloat16)
    gw = (_randn((E, d), 82, torch.float32) * d ** -0.5).bfloat16()
    bias = (0.05 * _randn((E,), 83, torch.float32))
    logits = (x.float() @ gw.float().t()).bfloat16()
    for _ in range(2):
        tok, experts, w, offs, inv, xs = ops.moe_gate_route(x.cuda(), gw.cuda(), bias.cuda(), K, identity_tail=tail,
                                                            gather=gather)
    ops.check_status()
    tok2, experts2, w2, offs2, inv2 = ops.moe_route(logits.cuda(), bias.cuda(), K, identity_tail=tail)
    n = T * K
    assert offs[-1].item() == n and torch.equal(offs, experts.bincount(minlength=E).cumsum(0).int())
    key = experts.long() * T + tok[:n].long()
    assert (key[1:] > key[:-1]).all()
    rows = inv.long().reshape(-1)
    assert torch.equal(tok[rows].view(T, K).long(), torch.arange(T, device="cuda").view(T, 1).expand(T, K))
    if tail:
        assert torch.equal(tok[n:], torch.arange(T, device="cuda", dtype=torch.int32))
    sel, sel2 = experts[rows].view(T, K), experts2[inv2.long().reshape(-1)].view(T, K)
    same = (sel == sel2).all(dim=1)
    assert same.float().mean().item() >= 0.97, same.float().mean().item()
    wa, wb = w[rows].view(T, K).float(), w2[inv2.long().reshape(-1)].view(T, K).float()
    assert (wa[same] - wb[same]).abs().max().item() <= 8e-3 if same.any() else True
    if gather:
        assert xs is not None and torch.equal(xs.cpu(), x[tok.cpu().long()])
    else:
        assert xs is None


# ----------------------------------------------------------------------------- head_dim 64 prefill, four heads per CTA
@pytest.mark.parametrize("Hq,Hkv", [(16, 4), (4, 1), (8, 1), (32, 8)])
def test_prefill_head_dim_64_four_heads_per_cta_matches_oracle(Hq, Hkv):
    """The tcgen05 kernel for head_dim 64 (four query heads of a KV head per CTA, 128-row tiles): ragged lengths
    around the tile and key-tile boundaries, with the plain grid and with the device-built tile list (bit-equal),
    against the CPU oracle."""
    ops, orc = _ops(), _oracle()
    D = 64
    assert ops.prefill_tile_rows(Hq, Hkv, D, D, torch.bfloat16) == 128
    lens = [540, 1, 127, 128, 129, 64, 65, 1000, 300, 63]
    T = sum(lens)
    q = _randn((T, Hq, D), 91, torch.bfloat16)
    k = _randn((T, Hkv, D), 92, torch.bfloat16)
    v = _randn((T, Hkv, D), 93, torch.bfloat16)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32)
    got = ops.prefill_varlen(q.cuda(), k.cuda(), v.cuda(), cu.cuda(), cu.cuda(), max(lens), max(lens), D ** -0.5)
    ops.check_status()
    want = orc.prefill_varlen(q, k, v, cu, cu, D ** -0.5)
    err = (got.float().cpu() - want).abs()
    assert err.max().item() <= 2e-2, err.max().item()
    assert (err.mean() / want.abs().mean()).item() <= 1e-2
    plan = ops.prefill_plan(cu.cuda(), T, max(lens), 128)
    again = ops.prefill_varlen(q.cuda(), k.cuda(), v.cuda(), cu.cuda(), cu.cuda(), max(lens), max(lens), D ** -0.5,
                               plan=plan)
    ops.check_status()
    assert torch.equal(again, got)
    # strided q / k / v (column slices of a fused projection), as the model passes them
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], dim=1).cuda()
    qs = qkv[:, :Hq * D].view(T, Hq, D)
    ks = qkv[:, Hq * D:(Hq + Hkv) * D].view(T, Hkv, D)
    vs = qkv[:, (Hq + Hkv) * D:].view(T, Hkv, D)
    strided = ops.prefill_varlen(qs, ks, vs, cu.cuda(), cu.cuda(), max(lens), max(lens), D ** -0.5)
    ops.check_status()
    assert torch.equal(strided, got)
