"""fp32 attention at head sizes 32 / 64 / 128: the tiled prompt kernel and the clustered decode kernel against the general kernels,
which take the same calls when the output does not start on a 16-byte boundary, over every form that both accept.

Bound: both sides add at most a few thousand fp32 products and weights below one, so they differ by far less than the 2e-5 that
fp32 kernels are held to against the oracle."""
import numpy as np
import pytest
import torch

from llm_from_scratch_b200.workloads import deal_blocks

pytestmark = pytest.mark.gpu
MAX_ABS = 2e-5


def _off_boundary(shape):
    n = int(np.prod(shape))
    return torch.zeros(n + 1, device="cuda")[1:].view(shape)


def _randn(seed, *shape):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).cuda()


def _cu(lens):
    return torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")


def _same(got, want):
    assert torch.isfinite(want).all() and (got - want).abs().max().item() <= MAX_ABS


# rows per CTA (32 / 64) follow from heads x tokens; lengths sit at the edges of tiles of 32 / 64 keys and of row tiles
@pytest.mark.parametrize("Hq,Hkv,D", [(4, 4, 32), (16, 4, 64), (6, 2, 64), (32, 8, 128), (8, 1, 128), (16, 4, 32)])
@pytest.mark.parametrize("lens", [[1], [33, 0, 64, 1, 65], [200, 31, 129, 127], [700, 641, 64, 3, 500]])
def test_packed_prompts(Hq, Hkv, D, lens):
    from llm_from_scratch_b200 import ops
    T, cu = sum(lens), _cu(lens)
    rows = _randn(1, T, (Hq + 2 * Hkv) * D)                       # views of one projection
    q, k, v = (x.unflatten(1, (-1, D)) for x in rows.split([Hq * D, Hkv * D, Hkv * D], 1))
    for sink in (None, _randn(2, Hq)):
        args = (q, k, v, cu, cu, max(lens), max(lens), D ** -0.5)
        want = ops.prefill_varlen(*args, out=_off_boundary((T, Hq, D)), sink=sink)
        _same(ops.prefill_varlen(*args, sink=sink), want)
    ops.check_status()


@pytest.mark.parametrize("page", [5, 16, 256])
@pytest.mark.parametrize("Hq,Hkv,D", [(16, 4, 64), (4, 2, 128), (16, 4, 32)])
def test_paged_prefix_and_blocks_outside_the_pool(page, Hq, Hkv, D):
    from llm_from_scratch_b200 import ops
    k_lens, q_lens = [700, 64, 65, 40, 3], [300, 64, 1, 17, 5]    # the last one: queries ahead of every key
    case = deal_blocks(k_lens, page, np.random.default_rng(0), pad_blocks=2)
    kc, vc = _randn(3, case.num_blocks, page, Hkv, D), _randn(4, case.num_blocks, page, Hkv, D)
    tables, q = torch.from_numpy(case.block_tables).cuda(), _randn(5, sum(q_lens), Hq, D)
    args = (q, None, None, _cu(q_lens), _cu(k_lens), max(q_lens), max(k_lens), D ** -0.5, kc, vc)
    want = ops.prefill_varlen(*args, tables, out=_off_boundary(q.shape))
    _same(ops.prefill_varlen(*args, tables), want)
    ops.check_status()
    bad = tables.clone()
    bad[0, 1], bad[1, 0] = case.num_blocks, -1                     # skipped and reported by both
    want = ops.prefill_varlen(*args, bad, out=_off_boundary(q.shape))
    assert ops.read_status_code() != 0
    _same(ops.prefill_varlen(*args, bad), want)
    assert ops.read_status_code() != 0


@pytest.mark.parametrize("Hq,Hkv,D", [(16, 4, 64), (16, 16, 128), (16, 16, 32)])
@pytest.mark.parametrize("n", [1, 70])
@pytest.mark.parametrize("q_len,prefix", [(1, 0), (1, 30), (2, 127), (3, 62), (8, 0), (8, 24), (9, 0)])
def test_short_portions(Hq, Hkv, D, n, q_len, prefix):
    """Sizes on both sides of the line between tiles and a warp per row; the other side is always the warp per row."""
    from llm_from_scratch_b200 import ops
    k_len = q_len + prefix
    case = deal_blocks([k_len] * n, 16, np.random.default_rng(n), pad_blocks=1)
    kc, vc = _randn(3, case.num_blocks, 16, Hkv, D), _randn(4, case.num_blocks, 16, Hkv, D)
    tables, q = torch.from_numpy(case.block_tables).cuda(), _randn(5, n * q_len, Hq, D)
    args = (q, None, None, _cu([q_len] * n), _cu([k_len] * n), q_len, k_len, D ** -0.5, kc, vc, tables)
    _same(ops.prefill_varlen(*args), ops.prefill_varlen(*args, out=_off_boundary(q.shape)))
    ops.check_status()


def test_more_sequences_than_a_grid_of_the_general_kernel_holds():
    from llm_from_scratch_b200 import ops
    n = 70000
    q, k, v, cu = _randn(1, n, 2, 32), _randn(2, n, 1, 32), _randn(3, n, 1, 32), torch.arange(n + 1, dtype=torch.int32, device="cuda")
    assert torch.equal(ops.prefill_varlen(q, k, v, cu, cu, 1, 1, 0.2), v.expand(n, 2, 32))
    ops.check_status()


def test_values_a_row_does_not_see_stay_out_of_it():
    from llm_from_scratch_b200 import ops
    lens, Hq, Hkv, D = [100, 90], 8, 2, 64
    cu, q, k, v = _cu(lens), _randn(6, 190, Hq, D), _randn(7, 190, Hkv, D), _randn(8, 190, Hkv, D)
    want = ops.prefill_varlen(q, k, v, cu, cu, 100, 100, 0.125)
    v[70, 0, 3], v[150, 1, 7], k[80, 1, 5] = float("inf"), float("nan"), float("inf")
    got = ops.prefill_varlen(q, k, v, cu, cu, 100, 100, 0.125)
    for lo, hi, heads in ((0, 70, slice(0, 4)), (0, 80, slice(4, 8)), (100, 190, slice(0, 4)), (100, 150, slice(4, 8))):
        assert torch.equal(got[lo:hi, heads], want[lo:hi, heads])
    assert not torch.isfinite(got[70:100, :4, 3]).any() and not torch.isfinite(got[150:, 4:, 7]).any()


# clusters of 8, 4, 2 and 1 CTAs per context follow from batch x heads and the length of the block table
@pytest.mark.parametrize("page", [1, 16, 48])
@pytest.mark.parametrize("Hq,Hkv,D,lens", [
    (16, 4, 64, [700]), (4, 4, 32, [1, 0, 7, 8, 9, 300]), (6, 2, 128, [33, 500, 16]), (32, 8, 128, [100, 900] * 8),
    (16, 4, 64, [2, 0, *range(1, 130, 2)]), (8, 1, 64, [63, 64, 65] * 40), (3, 1, 32, [400] * 300), (16, 16, 32, [16, 3, 9] * 50),
    (16, 4, 64, [8, 1, 5])])
def test_decode(page, Hq, Hkv, D, lens):
    from llm_from_scratch_b200 import ops
    case = deal_blocks(lens, page, np.random.default_rng(1), pad_blocks=2)
    kc, vc = _randn(9, case.num_blocks, page, Hkv, D), _randn(10, case.num_blocks, page, Hkv, D)
    q, tables, ctx = _randn(11, len(lens), Hq, D), torch.from_numpy(case.block_tables).cuda(), torch.from_numpy(case.context_lens).cuda()
    for sink in (None, _randn(12, Hq)):
        args = (q, kc, vc, tables, ctx, D ** -0.5)
        want = ops.paged_decode_gqa(*args, out=_off_boundary(q.shape), sink=sink)
        _same(ops.paged_decode_gqa(*args, sink=sink), want)
    ops.check_status()
    tables[0, 0] = case.num_blocks + 3
    want = ops.paged_decode_gqa(*args, out=_off_boundary(q.shape))
    assert ops.read_status_code() != 0
    _same(ops.paged_decode_gqa(*args), want)
    assert ops.read_status_code() != 0


def test_decode_calls_share_nothing():
    """Two streams, each with calls of its own in flight, give what one gives alone."""
    from llm_from_scratch_b200 import ops
    case = deal_blocks([900, 20, 400], 16, np.random.default_rng(2))
    kc, vc = _randn(13, case.num_blocks, 16, 4, 64), _randn(14, case.num_blocks, 16, 4, 64)
    tables, ctx = torch.from_numpy(case.block_tables).cuda(), torch.from_numpy(case.context_lens).cuda()
    qs = [_randn(15 + i, 3, 16, 64) for i in range(2)]
    want = [ops.paged_decode_gqa(q, kc, vc, tables, ctx, 0.125) for q in qs]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in qs], [[], []]
    for _ in range(20):
        for i, st in enumerate(streams):
            with torch.cuda.stream(st):
                got[i].append(ops.paged_decode_gqa(qs[i], kc, vc, tables, ctx, 0.125))
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for outs, w in zip(got, want) for g in outs)
