"""Kernels that start beside the launch before them: each pair against the same calls one behind the other, eager and captured.
The programs are equal, so the results are the same bits."""
import numpy as np
import pytest
import torch

from llm_from_scratch_b200.workloads import deal_blocks

pytestmark = pytest.mark.gpu


def _randn(seed, *shape):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).cuda()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("with_plan", [False, True])
@pytest.mark.parametrize("Hq,Hkv,D", [(16, 4, 64), (32, 8, 128)])
@pytest.mark.parametrize("lens", [[1, 17], [700, 1, 64, 900], [40] * 200])
def test_prompt_attention_beside_its_scatter(Hq, Hkv, D, lens, with_plan, captured):
    """The rows come straight from the launch before the call, and a decode over the rows that it scatters follows at once.  The
    attention of short prompts ends before the scatter of many rows, that of long ones behind it."""
    from llm_from_scratch_b200 import ops
    case, T, page, dt = deal_blocks(lens, 16, np.random.default_rng(D), pad_blocks=2), sum(lens), 16, torch.bfloat16
    slots = np.concatenate([case.block_tables[i, np.arange(n) // page].astype(np.int64) * page + np.arange(n) % page
                            for i, n in enumerate(lens)])
    slots = torch.from_numpy(slots).cuda()
    tables, ctx = torch.from_numpy(case.block_tables).cuda(), torch.from_numpy(case.context_lens).cuda()
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    sources = [_randn(i, T, (Hq + 2 * Hkv) * D).to(dt) for i in range(3)]
    rows, q1 = torch.zeros_like(sources[0]), _randn(9, len(lens), Hq, D).to(dt)
    q, k, v = (x.unflatten(1, (-1, D)) for x in rows.split([Hq * D, Hkv * D, Hkv * D], 1))
    pools = [torch.empty(case.num_blocks, page, Hkv, D, dtype=dt, device="cuda") for _ in range(2)]
    plan = ops.prefill_plan(cu, T, max(lens), ops.prefill_tile_rows(Hq, Hkv, D, D, dt)) if with_plan else None
    args = (cu, cu, max(lens), max(lens), D ** -0.5)
    outs = torch.empty(T, Hq, D, dtype=dt, device="cuda"), torch.empty_like(q1)

    def step():
        ops.prefill_varlen(q, k, v, *args, pools[0], pools[1], out=outs[0], plan=plan, slot_mapping=slots)
        ops.paged_decode_gqa(q1, *pools, tables, ctx, D ** -0.5, out=outs[1])

    graph = None
    for source in sources:
        rows.copy_(source)
        for p in pools:
            p.fill_(50.0)
        want = [ops.prefill_varlen(q, k, v, *args, plan=plan)]
        ops.store_kvcache(k, v, *pools, slots)
        torch.cuda.synchronize()
        want += [ops.paged_decode_gqa(q1, *pools, tables, ctx, D ** -0.5), *(p.clone() for p in pools)]
        rows.zero_()
        for p in pools:
            p.fill_(50.0)
        torch.cuda.synchronize()
        if captured and graph is None:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                step()
        rows.copy_(source)
        if captured:
            graph.replay()
        else:
            step()
        ops.check_status()
        assert all(torch.equal(a, b) for a, b in zip([*outs, *pools], want))


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("T,E,top,k,n,shared", [(2000, 16, 2, 1024, 704, True), (600, 8, 2, 256, 264, False), (1500, 32, 2, 2048, 1024, True)])
def test_expert_products_of_prompts_started_early(T, E, top, k, n, shared, captured):
    """Route, gather, up, down: both products may set up beside the launch before them."""
    from llm_from_scratch_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T)
    sets = E + 1 if shared else E
    up, down = ((torch.randn(sets, *s, generator=g, device="cuda") * s[1] ** -0.5).bfloat16() for s in ((2 * n, k), (k, n)))
    bias, x = torch.zeros(E, device="cuda"), torch.empty(T, k, dtype=torch.bfloat16, device="cuda")
    gate = torch.randn(k, E, generator=g, device="cuda").bfloat16()

    def layer(early):
        tok, _, _, offs, _ = ops.moe_route((x @ gate).contiguous(), bias, top, identity_tail=shared)
        dense = T if shared else 0
        act = ops.moe_grouped_gemm(x.index_select(0, tok), up, offs, None, swiglu=True, dense_rows=dense, early_launch=early)
        return ops.moe_grouped_gemm(act, down, offs, None, dense_rows=dense, early_launch=early)

    graph = None
    for _ in range(4):
        x.copy_(torch.randn(T, k, generator=g, device="cuda"))
        want = layer(False)
        torch.cuda.synchronize()
        if captured and graph is None:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                got = layer(True)
        if captured:
            graph.replay()
        else:
            got = layer(True)
        ops.check_status()
        assert torch.equal(got, want)
