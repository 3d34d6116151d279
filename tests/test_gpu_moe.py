"""Parity of the router, the token->expert permutation and the fused expert GEMMs with the CPU
oracle."""
import numpy as np
import pytest
import torch

from oracle import awq_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-2


@pytest.fixture(scope="module")
def A(built_library):
    import awq_b200
    assert torch.cuda.is_available()
    return awq_b200


@pytest.mark.parametrize("t,e,k,renorm,dtype", [
    (1, 128, 8, True, torch.float32), (16, 128, 8, True, torch.float32),
    (333, 128, 8, False, torch.float32), (7, 8, 2, True, torch.float16),
    (5, 1000, 32, True, torch.float32), (4096, 128, 8, True, torch.float32),
])
def test_topk_softmax(A, t, e, k, renorm, dtype):
    g = torch.randn(t, e, generator=torch.Generator().manual_seed(t + e)).to(dtype)
    hs = torch.empty(t, 4, dtype=torch.float16, device="cuda")
    w, ids, tok = A.fused_topk(hs, g.cuda(), k, renorm)
    rw, rids, rtok = O.topk_softmax(g.float().numpy(), k, renorm)
    assert np.array_equal(ids.cpu().numpy(), rids)          # indices bit-exact
    assert np.array_equal(tok.cpu().numpy(), rtok)
    assert np.allclose(w.cpu().numpy(), rw, rtol=2e-5, atol=1e-7)


def test_topk_ties_pick_lower_id(A):
    g = torch.zeros(3, 128)
    g[1, 100] = 1.0
    hs = torch.empty(3, 4, dtype=torch.float16, device="cuda")
    _, ids, _ = A.fused_topk(hs, g.cuda(), 8, True)
    assert ids[0].tolist() == list(range(8))
    assert ids[1].tolist() == [100] + list(range(7))


@pytest.mark.parametrize("t,k,e,blk", [
    (1, 8, 128, 16), (16, 8, 128, 16), (128, 8, 128, 16), (1024, 8, 128, 16), (4096, 8, 128, 16),
    (4, 3, 4, 4), (33, 2, 8, 4), (100, 1, 1000, 8), (64, 8, 128, 64),
])
def test_moe_align_bit_exact(A, t, k, e, blk):
    rng = np.random.default_rng(t * 31 + e)
    ids = np.stack([rng.permutation(e)[:k] for _ in range(t)]).astype(np.int32)
    s, eid, post = A.moe_align_block_size(torch.from_numpy(ids).cuda(), blk, e)
    rs, reid, rpost = O.moe_align_block_size(ids, blk, e)
    assert np.array_equal(post.cpu().numpy(), rpost)
    assert np.array_equal(s.cpu().numpy(), rs)
    assert np.array_equal(eid.cpu().numpy(), reid)


# Around the length from which clusters build the histogram together: whole and ragged eighths, one
# expert, the most experts, experts of other ranks.
@pytest.mark.parametrize("t,k,e,blk", [(256, 8, 128, 16), (2049, 1, 1, 8), (257, 8, 1024, 8),
                                       (683, 3, 60, 128), (4099, 7, 128, 128)])
def test_moe_align_long_lists(A, t, k, e, blk):
    rng = np.random.default_rng(t)
    ids = rng.integers(0, e, size=(t, k)).astype(np.int32)
    emap = np.arange(e, dtype=np.int32)
    emap[1::3] = -1
    for m in (None, emap):
        s, eid, post = A.moe_align_block_size(torch.from_numpy(ids).cuda(), blk, e,
                                              None if m is None else torch.from_numpy(m).cuda(),
                                              ignore_invalid_experts=m is not None)
        want = O.moe_align_block_size(ids, blk, e) if m is None else O.moe_align_block_size(ids, blk, e, m)
        for got, ref in zip((s, eid, post), want):
            got, ref = got.cpu().numpy().ravel(), np.asarray(ref).ravel()
            np.testing.assert_array_equal(got[:len(ref)], ref)


def test_moe_align_docstring_example(A, golden):
    ids = torch.from_numpy(golden["align.topk_ids"]).cuda()
    s, eid, post = A.moe_align_block_size(ids, 4, 4)
    assert post.item() == 16
    assert s[:16].cpu().tolist() == golden["align.sorted_ids"].tolist()
    assert eid[:4].cpu().tolist() == [0, 1, 2, 3]


def test_moe_align_expert_map(A):
    rng = np.random.default_rng(9)
    t, k, e, blk = 50, 4, 16, 8
    ids = np.stack([rng.permutation(e)[:k] for _ in range(t)]).astype(np.int32)
    emap = np.full(e, -1, dtype=np.int32)
    emap[4:8] = np.arange(4)
    s, eid, post = A.moe_align_block_size(torch.from_numpy(ids).cuda(), blk, e,
                                          torch.from_numpy(emap).cuda(),
                                          ignore_invalid_experts=True)
    rs, reid, rpost = O.moe_align_block_size(ids, blk, e, emap)
    assert np.array_equal(post.cpu().numpy(), rpost)
    assert np.array_equal(s.cpu().numpy(), rs)
    assert np.array_equal(eid.cpu().numpy(), reid)


def test_moe_align_against_installed_vllm(A):
    try:
        from vllm.model_executor.layers.fused_moe.moe_align_block_size import (
            moe_align_block_size as v_align)
        import vllm._moe_C  # noqa: F401
    except Exception as e:  # pragma: no cover
        pytest.skip(f"vllm compiled ops unavailable: {e}")
    rng = np.random.default_rng(4)
    t, k, e, blk = 200, 8, 128, 16
    ids = np.stack([rng.permutation(e)[:k] for _ in range(t)]).astype(np.int32)
    idt = torch.from_numpy(ids).cuda()
    s, eid, post = A.moe_align_block_size(idt, blk, e)
    vs, veid, vpost = v_align(idt, blk, e)
    assert post.item() == vpost.item()
    nb = post.item() // blk
    assert torch.equal(eid[:nb], veid[:nb])
    # same set of pairs per expert; the order inside an expert's run is ours (ascending)
    a = s[:post.item()].cpu().numpy().reshape(nb, blk)
    b = vs[:post.item()].cpu().numpy().reshape(nb, blk)
    ee = eid[:nb].cpu().numpy()
    for x in np.unique(ee):
        assert sorted(a[ee == x].reshape(-1).tolist()) == sorted(b[ee == x].reshape(-1).tolist())


def _moe_case(e, h, i, t, k, seed):
    from awq_b200 import synth
    w1, w2 = synth.moe_layer_tensors(e, h, i, 128, seed=seed)
    x = synth.activations(t, h, seed=seed + 1)
    logits = synth.gating_logits(t, e, seed=seed + 2)
    return w1, w2, x, logits


@pytest.mark.parametrize("e,h,i,t,k", [
    (4, 256, 128, 5, 2), (8, 512, 256, 1, 2), (16, 2048, 768, 16, 8), (128, 2048, 768, 1, 8),
    (128, 2048, 768, 40, 8), (8, 256, 128, 300, 2), (8, 512, 256, 777, 2),
    (128, 2048, 768, 128, 8), (128, 2048, 768, 1024, 8), (128, 2048, 768, 4096, 8),
    # 8-row blocks with experts that need several blocks, and 16-row blocks
    (16, 512, 256, 60, 2), (128, 2048, 768, 200, 8), (8, 256, 128, 50, 2),
])
def test_fused_experts_vs_oracle(A, e, h, i, t, k):
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=e + t)
    w, ids, _ = O.topk_softmax(logits.numpy(), k, True)
    ref = O.fused_experts_fp32(x.numpy(), *[a.numpy() for a in w1], *[a.numpy() for a in w2],
                               w, ids)
    w1d = tuple(a.cuda() for a in w1)
    w2d = tuple(a.cuda() for a in w2)
    y = A.fused_experts(x.cuda(), w1d, w2d, torch.from_numpy(w).cuda(),
                        torch.from_numpy(ids).cuda())
    torch.cuda.synchronize()
    y = y.cpu().numpy()
    err = O.rel_err(y, ref)
    assert err < TOL, f"rel err {err}"
    # whole layer through the router as well
    y2 = A.fused_moe(x.cuda(), w1d, w2d, logits.cuda(), k, True).cpu().numpy()
    assert O.rel_err(y2, ref) < TOL


@pytest.mark.parametrize("group", [128, 64])
@pytest.mark.parametrize("counts", [
    (0, 1, 129, 256, 257, 128, 17, 300),     # around the multiples of 128 rows, a gap
    (513, 0, 0, 0, 0, 0, 0, 15),             # three tiles of one expert, experts without rows
])
def test_prefill_tiles_per_expert(A, counts, group):
    """The tile table of the grouped GEMMs: experts with row counts at the edges of its entries."""
    from awq_b200 import synth
    e, h, i = len(counts), 512, 384
    ids = torch.cat([torch.full((c,), x, dtype=torch.int32) for x, c in enumerate(counts)])
    t = ids.numel()
    ids = ids[torch.randperm(t, generator=torch.Generator().manual_seed(t))].reshape(t, 1)
    w1, w2 = synth.moe_layer_tensors(e, h, i, group, seed=t + group)
    x = synth.activations(t, h, seed=t)
    w = torch.rand(t, 1, generator=torch.Generator().manual_seed(1)) + 0.5
    ref = O.fused_experts_fp32(x.numpy(), *[a.numpy() for a in w1], *[a.numpy() for a in w2],
                               w.numpy(), ids.numpy(), group)
    y = A.fused_experts(x.cuda(), tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2), w.cuda(),
                        ids.cuda(), group_size=group)
    torch.cuda.synchronize()
    # fp16 weights, intermediate activations, rows and output: 2^-11 each, far inside TOL
    assert O.rel_err(y.cpu().numpy(), ref) < TOL


# Every size of a tile above 128 rows, with row counts at its multiples, which do not fall on the 128-row blocks of
# the permutation, and shapes for which that size is taken (asserted); then counts that leave 128 rows or 160.
TILE_CASES = [
    (144, 1024, 1024, (143, 144, 145, 287, 289, 432, 575, 17)),
    (160, 768, 384, (159, 160, 161, 319, 321, 1, 17, 0, 119, 120, 121, 122, 123, 124, 125, 126)),
    (176, 768, 384, (175, 176, 177, 351, 353, 1, 17, 0, 116, 117, 118, 119, 120, 121, 122, 123)),
    (192, 768, 512, (191, 192, 193, 383, 385, 1, 17, 0, 132, 133, 134, 135, 136, 137, 139, 140)),
    (208, 1024, 512, (207, 208, 209, 415, 417, 1, 17, 0, 148, 149, 150, 151, 152, 153, 154, 155)),
    (224, 1792, 640, (223, 224, 225, 447, 449, 1, 17, 0, 150, 156)),
    (240, 2048, 1536, (239, 240, 241, 481, 17, 10)),
    (256, 4096, 2048, (255, 257, 241)), (256, 4096, 2048, (256, 511, 0)),
    (160, 1024, 1024, (159, 160, 161, 17, 319, 1, 209, 0)), (128, 1024, 1024, (191, 192, 193, 17, 383, 1, 271, 0)),
    (128, 1024, 1024, (207, 208, 209, 415, 0, 321, 1, 16)), (128, 1024, 1024, (223, 224, 225, 447, 0, 385, 1, 16)),
]


@pytest.mark.parametrize("group", [128, 64])
@pytest.mark.parametrize("rows,h,i,counts", TILE_CASES)
def test_prefill_tiles_between_the_blocks(A, rows, h, i, counts, group):
    from awq_b200 import _lib, synth
    e = len(counts)
    ids = torch.cat([torch.full((c,), x, dtype=torch.int32) for x, c in enumerate(counts)])
    t = ids.numel()
    assert _lib.load().awq_b200_moe_tile_rows(t, 1, e, e, h, i, 0) == rows
    ids = ids[torch.randperm(t, generator=torch.Generator().manual_seed(t))].reshape(t, 1)
    w1, w2 = synth.moe_layer_tensors(e, h, i, group, seed=t + group)
    x = synth.activations(t, h, seed=t)
    w = torch.rand(t, 1, generator=torch.Generator().manual_seed(1)) + 0.5
    ref = O.fused_experts_fp32(x.numpy(), *[a.numpy() for a in w1], *[a.numpy() for a in w2],
                               w.numpy(), ids.numpy(), group)
    y = A.fused_experts(x.cuda(), tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2), w.cuda(),
                        ids.cuda(), group_size=group)
    torch.cuda.synchronize()
    # fp16 weights, intermediate activations, rows and output: 2^-11 each, far inside TOL
    assert O.rel_err(y.cpu().numpy(), ref) < TOL


# Runs of row blocks that begin, end or go on at the 32nd and the 256th block, where the tile table's scan changes
# warps and starts again, and runs of one block there; 257 to 300 blocks in all.
@pytest.mark.parametrize("counts", [
    (31 * 128, 5, 1, 30 * 128 + 7, 128, 192 * 128, 1, 3, 129), (32 * 128 - 1, 224 * 128, 77, 0, 40 * 128 + 1),
    (255 * 128, 128, 1), (257 * 128,),
])
def test_prefill_tile_table_of_many_blocks(A, counts):
    from awq_b200 import synth
    e, h, i = len(counts), 256, 128
    ids = torch.cat([torch.full((c,), x, dtype=torch.int32) for x, c in enumerate(counts)])
    t = ids.numel()
    ids = ids[torch.randperm(t, generator=torch.Generator().manual_seed(t))].reshape(t, 1)
    w1, w2 = synth.moe_layer_tensors(e, h, i, 128, seed=t)
    x = synth.activations(t, h, seed=t)
    w = torch.rand(t, 1, generator=torch.Generator().manual_seed(1)) + 0.5
    ref = O.fused_experts_fp32(x.numpy(), *[a.numpy() for a in w1], *[a.numpy() for a in w2],
                               w.numpy(), ids.numpy(), 128)
    y = A.fused_experts(x.cuda(), tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2), w.cuda(), ids.cuda())
    torch.cuda.synchronize()
    # Row by row, as rows differ in size (silu(gate) * up has long tails).  Roundings of 2^-11 at most of the weights,
    # the activation, the row and the output, independent over the 256 and 128 terms of a sum: some 2^-11 of the
    # row's norm, 1 / 20 of TOL.  A row that no tile has, or another expert's tile, is off by all of itself.
    err = np.linalg.norm(y.cpu().numpy().astype(np.float32) - ref, axis=1)
    assert (err <= TOL * np.linalg.norm(ref, axis=1)).all()


# Groups of 128: gemm_ts; 64 and 32: the mma.sync kernels, whose down GEMM adds the slots itself unless its
# counters do not fit (64 tokens of 8192).  Every case has at least twice as many experts as pairs, or is
# not direct.
@pytest.mark.parametrize("group", [128, 64, 32])
@pytest.mark.parametrize("t,k,e,h,i", [(1, 8, 128, 2048, 768), (2, 8, 128, 2048, 768),
                                       (2, 4, 16, 512, 256), (1, 2, 8, 256, 128),
                                       (4, 8, 128, 2048, 768), (8, 8, 128, 2048, 768),
                                       (5, 8, 128, 8192, 256), (64, 1, 128, 8192, 256),
                                       (64, 1, 128, 512, 256)])
def test_direct_mode_for_a_handful_of_pairs_equals_the_permuted_path(A, t, k, e, h, i, group, monkeypatch):
    """A handful of (token, slot) pairs skip the permutation kernel (one row block per pair, experts read
    from topk_ids): the same roundings as through the permutation, on the mma.sync kernels the same bits.
    With an expert_map (here the identity) the direct mode reads the mapped ids."""
    from awq_b200 import ops, synth
    assert 2 * t * k <= e and t * k <= ops.MOE_DIRECT_MAX_PAIRS
    w1, w2 = synth.moe_layer_tensors(e, h, i, group, seed=40 + t)
    x, logits = synth.activations(t, h, seed=41 + t), synth.gating_logits(t, e, seed=42 + t)
    w1d = tuple(a.cuda() for a in w1)
    w2d = tuple(a.cuda() for a in w2)
    wts, ids, _ = A.fused_topk(x.cuda(), logits.cuda(), k, True)
    emap = torch.arange(e, dtype=torch.int32, device="cuda")

    def both(ids):
        direct = A.fused_experts(x.cuda(), w1d, w2d, wts, ids, group_size=group)
        mapped = A.fused_experts(x.cuda(), w1d, w2d, wts, ids, group_size=group, global_num_experts=e,
                                 expert_map=emap)
        with monkeypatch.context() as patch:
            patch.setattr(ops, "MOE_DIRECT_MAX_PAIRS", 0)
            permuted = A.fused_experts(x.cuda(), w1d, w2d, wts, ids, group_size=group)
        assert torch.equal(direct, mapped)
        if group != 128:
            assert torch.equal(direct, permuted)
        # gemm_ts cuts K by the number of tiles: fp32 sums in another order, which put some values on the
        # other side of a rounding.  2^-11 each, fewer than one in six.
        diff = (direct.double() - permuted.double()).norm() / permuted.double().norm()
        assert diff < 2e-4
        return direct

    both(ids)
    # two slots of one token on the same expert: the pair blocks stay independent
    if k == 1:
        return
    ids2 = ids.clone()
    ids2[:, 1] = ids2[:, 0]
    direct2 = both(ids2)
    ref = O.fused_experts_fp32(x.numpy(), *[a.numpy() for a in w1], *[a.numpy() for a in w2],
                               wts.cpu().numpy(), ids2.cpu().numpy(), group)
    assert O.rel_err(direct2.float().cpu().numpy(), ref) < TOL


# Expert GEMMs of small batches: one tile shared by many CTAs, one unit of K in all, column slabs past
# the edge (H an odd multiple of 128), 8- and 16-row blocks with several blocks per expert, direct mode
# at its smallest and largest, tiles of several 16-row blocks (the last two); with experts of another
# rank (every third id) absent.
@pytest.mark.parametrize("t,k,e,h,i", [(1, 1, 8, 128, 128), (1, 8, 64, 1152, 384), (8, 8, 128, 512, 640),
                                       (9, 8, 128, 384, 128), (35, 4, 12, 2048, 384),
                                       (72, 4, 16, 640, 256), (70, 2, 8, 640, 256)])
@pytest.mark.parametrize("parallel", [False, True])
def test_small_batch_experts_edges(A, t, k, e, h, i, parallel):
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=t + e)
    w, ids, _ = O.topk_softmax(logits.numpy(), k, True)
    here = np.array([n for n in range(e) if not parallel or n % 3 != 1])
    emap = np.full(e, -1, dtype=np.int32)
    emap[here] = np.arange(len(here))
    # the oracle sees absent pairs as pairs of weight zero
    w_ref = np.where(emap[ids] >= 0, w, 0).astype(np.float32)
    ref = O.fused_experts_fp32(x.numpy(), *[a.numpy() for a in w1], *[a.numpy() for a in w2], w_ref, ids)
    local = [tuple(a[torch.from_numpy(here)].contiguous().cuda() for a in ws) for ws in (w1, w2)]
    y = A.fused_experts(x.cuda(), *local, torch.from_numpy(w).cuda(), torch.from_numpy(ids).cuda(),
                        global_num_experts=e,
                        expert_map=torch.from_numpy(emap).cuda() if parallel else None)
    torch.cuda.synchronize()
    y = y.cpu().numpy()
    assert np.isfinite(y.astype(np.float32)).all()
    # fp16 intermediate activations, rows and output: 2^-11 each, far inside TOL
    if np.abs(ref).max() == 0:
        assert not y.any()
    else:
        assert O.rel_err(y, ref) < TOL


# One or two tokens: gate_up on clusters (units of gate and up that do not divide by them, an edge of the columns inside
# a slab, one unit in all) or in ranges, down on clusters of a token's slots; every number of slots; a third of the experts absent.
@pytest.mark.parametrize("t,k,h,i", [(1, 2, 256, 128), (1, 3, 1152, 384), (1, 4, 4096, 1536), (1, 5, 640, 640),
                                     (1, 6, 2048, 768), (1, 7, 896, 896), (1, 8, 2048, 1024), (2, 4, 2048, 768),
                                     (2, 3, 512, 128), (1, 1, 2048, 768), (1, 2, 2048, 256), (2, 1, 256, 128)])
@pytest.mark.parametrize("parallel", [False, True])
def test_direct_clusters_round_like_the_permuted_path(A, t, k, h, i, parallel, monkeypatch):
    from awq_b200 import ops
    e = 64
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=t + k)
    w, ids, _ = A.fused_topk(x.cuda(), logits.cuda(), k, True)
    here = torch.tensor([n for n in range(e) if not parallel or n % 3 != 1])
    emap = torch.full((e,), -1, dtype=torch.int32)
    emap[here] = torch.arange(len(here), dtype=torch.int32)
    local = [tuple(a[here].contiguous().cuda() for a in ws) for ws in (w1, w2)]
    kwargs = dict(global_num_experts=e, expert_map=emap.cuda() if parallel else None)
    y = [A.fused_experts(x.cuda(), *local, w, ids, **kwargs) for _ in range(3)]
    with monkeypatch.context() as patch:
        patch.setattr(ops, "MOE_DIRECT_MAX_PAIRS", 0)
        permuted = A.fused_experts(x.cuda(), *local, w, ids, **kwargs)
    torch.cuda.synchronize()
    assert torch.equal(y[0], y[1]) and torch.equal(y[0], y[2])
    # fp32 sums in another order put some values on the other side of a rounding: 2^-11 each, fewer than one in six
    assert (y[0].double() - permuted.double()).norm() <= 2e-4 * permuted.double().norm()


# Tokens of one expert each: whole prompts (grouped tiles), a server's batch (a tile per row block).
@pytest.mark.parametrize("t,e", [(300, 4), (40, 8)])
def test_rows_leave_the_range_of_fp16_only_before_their_weight(A, t, e):
    """Rows of the down projection beyond 65504 whose routed weight brings them back: the weight is
    applied in fp32, ahead of the rounding to fp16."""
    h, i, k = 512, 256, 2
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=t)
    _, ids, _ = O.topk_softmax(logits.numpy(), k, True)
    one = np.ones((t, k), dtype=np.float32)
    rows = O.fused_experts_fp32(x.numpy(), *[a.numpy() for a in w1], *[a.numpy() for a in w2], one, ids)
    # row sums far beyond 65504, the weighted ones (by 2^-6, exact) inside
    w2 = (w2[0], w2[1] * float(2 ** np.round(np.log2(4e5 / np.abs(rows).max()))), w2[2])
    w = one * 2.0 ** -6
    ref = O.fused_experts_fp32(x.numpy(), *[a.numpy() for a in w1], *[a.numpy() for a in w2], w, ids)
    assert 2 ** 6 * np.abs(ref).max() > 2 * 65504 and np.abs(ref).max() < 30000
    y = A.fused_experts(x.cuda(), tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2),
                        torch.from_numpy(w).cuda(), torch.from_numpy(ids).cuda()).float().cpu().numpy()
    assert np.isfinite(y).all()
    assert O.rel_err(y, ref) < TOL


# Grouped tiles (75 rows per expert and slot; no tile is split along K), and the direct mode (a unit of K
# per CTA in all of its calls, so that their sums have one order).
@pytest.mark.parametrize("t,e,h,i,k", [(300, 4, 512, 384, 2), (1, 16, 512, 384, 8), (2, 16, 512, 384, 4)])
def test_a_slot_is_rounded_once_weighted_and_then_added(A, t, e, h, i, k):
    """Every (token, slot) row is rounded to fp16 after its routed weight and a token's rows are added
    in fp32: the output is the rounded sum of what the slots give one by one, bit for bit."""
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=7 * t)
    w1d, w2d, xd = tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2), x.cuda()
    w, ids, _ = A.fused_topk(xd, logits.cuda(), k, True)
    y = A.fused_experts(xd, w1d, w2d, w, ids)
    total = torch.zeros(t, h, device="cuda")
    for s in range(k):
        total += A.fused_experts(xd, w1d, w2d, w[:, s:s + 1].contiguous(), ids[:, s:s + 1].contiguous()).float()
    assert torch.equal(y, total.half())


# Rows per expert on average: 5, 9, 15, 25, 35.
@pytest.mark.parametrize("group", [128, 64])
@pytest.mark.parametrize("t", [20, 36, 60, 100, 140])
def test_batches_below_prefill_apply_the_scales_in_fp32(A, t, group):
    """Below 36 rows per expert the error against 64 bits is that of the roundings of activations, rows and
    output, which weights rounded to (q - z) * s would exceed by a third."""
    from awq_b200 import synth
    e, h, i, k = 8, 512, 256, 2
    w1, w2 = synth.moe_layer_tensors(e, h, i, group, seed=t)
    x, logits = synth.activations(t, h, seed=t + 1), synth.gating_logits(t, e, seed=t + 2)
    w, ids, _ = O.topk_softmax(logits.numpy(), k, True)
    y = A.fused_experts(x.cuda(), tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2),
                        torch.from_numpy(w).cuda(), torch.from_numpy(ids).cuda(), group_size=group)

    def layer(r):  # in 64 bits, r at the places where the kernels round
        out = np.zeros((t, h))
        for n in range(e):
            tok, slot = np.nonzero(ids == n)
            m1, m2 = (O.dequantize_fp32(*[a[n].numpy() for a in ws], group).astype(np.float64) for ws in (w1, w2))
            gu = x.double().numpy()[tok] @ m1
            act = r(gu[:, :i] / (1 + np.exp(-gu[:, :i])) * gu[:, i:])
            np.add.at(out, tok, r(act @ m2 * w[tok, slot, None]))
        return r(out)

    exact = layer(lambda v: v)
    rounded = np.linalg.norm(layer(lambda v: v.astype(np.float16).astype(np.float64)) - exact)
    # 10 %: another set of the same roundings (fp32 sums, __expf), 10^4 values and more
    assert np.linalg.norm(y.double().cpu().numpy() - exact) < 1.1 * rounded


def test_prefill_ids_of_no_expert_contribute_nothing(A):
    """Without an expert_map the permutation drops ids outside [0, E) (padding tokens carry -1): such a
    (token, slot) pair adds zero, whatever earlier calls left in the scratch."""
    e, h, i, t, k = 8, 512, 256, 500, 2
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=17)
    w1d, w2d = tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2)
    w, ids, _ = O.topk_softmax(logits.numpy(), k, True)
    # a larger batch first: its entries, rows beyond the next call's among them, stay in the scratch
    wl, il = (torch.from_numpy(np.tile(a, (4, 1))).cuda() for a in (w, ids))
    A.fused_experts(torch.full((4 * t, h), 3e4, dtype=torch.float16, device="cuda"), w1d, w2d, wl, il)
    rng = np.random.default_rng(5)
    some = ids.copy()
    some[rng.random((t, k)) < 0.3] = -1
    some[rng.random((t, k)) < 0.1] = e
    some[7] = -1
    w_ref = np.where((some >= 0) & (some < e), w, 0).astype(np.float32)
    ref = O.fused_experts_fp32(x.numpy(), *[a.numpy() for a in w1], *[a.numpy() for a in w2], w_ref, ids)
    y = A.fused_experts(x.cuda(), w1d, w2d, torch.from_numpy(w).cuda(), torch.from_numpy(some).cuda())
    y = y.float().cpu().numpy()
    assert not y[7].any()
    assert np.isfinite(y).all() and O.rel_err(y, ref) < TOL


def test_wna16_layout_converts_back_bit_exact(A, golden):
    """uint8 [E, N, K/2] (vLLM's MoE WNA16 layout) -> AWQ layout on the device: vLLM's own
    converted tensors give back the AWQ tensors they were made from, and stacked random experts
    agree with the oracle's conversion."""
    import os
    g = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden",
                             "wna16_golden.npz"))
    for name in ("small", "wide", "g64"):
        grp = int(g[f"{name}.group"][0])
        q, s, z = A.wna16_to_awq(torch.from_numpy(g[f"{name}.wna16_qweight"])[None].cuda(),
                                 torch.from_numpy(g[f"{name}.wna16_scales"])[None].cuda(),
                                 torch.from_numpy(g[f"{name}.wna16_qzeros"])[None].cuda(), grp)
        assert np.array_equal(q[0].cpu().numpy(), g[f"{name}.qweight"])
        assert np.array_equal(z[0].cpu().numpy(), g[f"{name}.qzeros"])
        assert np.array_equal(s[0].cpu().numpy(), g[f"{name}.scales"])
    w1, w2, _, _ = _moe_case(6, 384, 160, 1, 2, seed=3)     # ragged tiles: N = 320 / 384, K = 384 / 160
    for qw, sc, qz in (w1, w2):
        wu = np.stack([O.awq_to_wna16_qweight(a) for a in qw.numpy()])
        zu = np.stack([O.awq_to_wna16_qzeros(a) for a in qz.numpy()])
        su = np.ascontiguousarray(sc.numpy().transpose(0, 2, 1))
        grp = qw.shape[1] // sc.shape[1]
        q, s, z = A.wna16_to_awq(torch.from_numpy(wu).cuda(), torch.from_numpy(su).cuda(),
                                 torch.from_numpy(zu).cuda(), grp)
        assert torch.equal(q.cpu(), qw) and torch.equal(z.cpu(), qz) and torch.equal(s.cpu(), sc)


def test_fused_experts_accepts_the_reference_call_form(A):
    """w1 / w2 as the stacked qweight tensors plus a quant_config object carrying scales and zero
    points (vLLM fused_moe.py:1587-1599) gives the same bits as the triple form."""
    from types import SimpleNamespace
    e, h, i, t, k = 16, 512, 256, 33, 4
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=5)
    w1d = tuple(a.cuda() for a in w1)
    w2d = tuple(a.cuda() for a in w2)
    wts, ids, _ = A.fused_topk(x.cuda(), logits.cuda(), k, True)
    y = A.fused_experts(x.cuda(), w1d, w2d, wts, ids)
    qc = SimpleNamespace(w1_scale=w1d[1], w2_scale=w2d[1], w1_zp=w1d[2], w2_zp=w2d[2],
                         block_shape=[0, 128])
    y2 = A.fused_experts(x.cuda(), w1d[0], w2d[0], wts, ids, quant_config=qc)
    assert torch.equal(y, y2)
    with pytest.raises(ValueError):
        A.fused_experts(x.cuda(), w1d[0], w2d[0], wts, ids)
    with pytest.raises(ValueError):
        A.fused_experts(x.cuda(), w1d[0], w2d[0], wts, ids,
                        quant_config=SimpleNamespace(w1_scale=w1d[1], w2_scale=w2d[1],
                                                     w1_zp=None, w2_zp=None))


@pytest.mark.parametrize("t", [20, 400])
def test_fused_experts_expert_parallel_shards_sum(A, t):
    """Two expert-parallel shards (expert_map) add up to the unsharded layer (T = 20: streaming
    kernels, T = 400: grouped tcgen05 GEMMs with blocks of experts that live on another rank)."""
    e, h, i, k = 8, 256, 128, 2
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=77)
    w, ids, _ = O.topk_softmax(logits.numpy(), k, True)
    wt, idt = torch.from_numpy(w).cuda(), torch.from_numpy(ids).cuda()
    full = A.fused_experts(x.cuda(), tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2),
                           wt, idt).float()
    acc = torch.zeros_like(full)
    for lo in (0, 4):
        emap = torch.full((e,), -1, dtype=torch.int32)
        emap[lo:lo + 4] = torch.arange(4, dtype=torch.int32)
        w1s = tuple(a[lo:lo + 4].contiguous().cuda() for a in w1)
        w2s = tuple(a[lo:lo + 4].contiguous().cuda() for a in w2)
        acc += A.fused_experts(x.cuda(), w1s, w2s, wt, idt, global_num_experts=e,
                               expert_map=emap.cuda()).float()
    assert O.rel_err(acc.cpu().numpy(), full.cpu().numpy()) < 5e-3


def test_expert_parallel_batch_takes_the_kernels_of_its_rows_per_expert(A):
    """64 tokens on one of eight ranks are four rows per expert however few experts live here: the calls
    below prefill run the same kernels with and without an expert_map."""
    from torch.profiler import ProfilerActivity, profile
    e, h, i, t, k = 128, 512, 256, 64, 8
    w1, w2, x, logits = _moe_case(16, h, i, t, 8, seed=3)
    w1d, w2d, xd = tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2), x.cuda()
    logits = torch.randn(t, e, generator=torch.Generator().manual_seed(4)).cuda()
    w, ids, _ = A.fused_topk(xd, logits, k, True)
    emap = torch.full((e,), -1, dtype=torch.int32, device="cuda")
    emap[32:48] = torch.arange(16, dtype=torch.int32, device="cuda")

    def call():
        return A.fused_experts(xd, w1d, w2d, w, ids, global_num_experts=e, expert_map=emap)

    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    names = [event.key for event in prof.key_averages() if "awq::" in event.key]
    if not names:
        pytest.skip("the profiler sees no kernels here")
    assert any("gemm_ts_kernel" in n for n in names), names
    assert not any("gemm_wt_kernel" in n for n in names), names


# Up to three tiles, for which clusters of more than eight CTAs would be estimated best, and more; ranges with many units.
@pytest.mark.parametrize("k,h,i,clusters", [(1, 2048, 768, 1), (2, 2048, 256, 1), (1, 1024, 384, 1), (8, 640, 640, 1),
                                            (8, 2048, 768, 0)])
def test_one_token_runs_gate_up_on_clusters(A, k, h, i, clusters):
    w1, w2, x, logits = _moe_case(16, h, i, 1, k, seed=3)
    w1d, w2d, xd = tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2), x.cuda()
    w, ids, _ = A.fused_topk(xd, logits.cuda(), k, True)
    A.fused_experts(xd, w1d, w2d, w, ids)
    torch.cuda.synchronize()
    forms = _ts_forms(lambda: A.fused_experts(xd, w1d, w2d, w, ids))
    if not forms:
        pytest.skip("the profiler sees no kernels here")
    assert [f[3] for f in forms if f[:3] == (4, 1, 128)] == [clusters], forms


def test_fused_moe_full_size_rows_are_independent(A):
    """Benchmark-size check without the oracle: a token's output does not depend on which other
    tokens share the batch, so the first rows of the T = 4096 layer (tcgen05 grouped GEMMs)
    must match the same tokens run as a T = 48 batch (weight-streaming kernels)."""
    e, h, i, k = 128, 2048, 768, 8
    w1, w2, x, logits = _moe_case(e, h, i, 4096, k, seed=123)
    w1d = tuple(a.cuda() for a in w1)
    w2d = tuple(a.cuda() for a in w2)
    big = A.fused_moe(x.cuda(), w1d, w2d, logits.cuda(), k, True)
    small = A.fused_moe(x[:48].cuda().contiguous(), w1d, w2d, logits[:48].cuda().contiguous(), k, True)
    torch.cuda.synchronize()
    assert torch.isfinite(big.float()).all()
    assert O.rel_err(big[:48].cpu().numpy(), small.float().cpu().numpy()) < 5e-3


@pytest.mark.parametrize("t,h,i,e,k", [(1, 2048, 768, 128, 8), (16, 2048, 768, 128, 8),
                                       (8, 256, 128, 50, 2), (40, 512, 256, 12, 2),
                                       (256, 2048, 768, 128, 8), (300, 512, 256, 4, 2)])
def test_experts_on_decode_layout_copies_equal_checkpoint_layout(A, t, h, i, e, k):
    """Decode-layout copies of the expert weights.  fused_experts accepts them and reads the checkpoint
    layout; the C ABI reads them when told so (flag bit 1): bit-identical to the same mma.sync kernels on
    the checkpoint layout, which run when the scratch has no room for partial tiles."""
    from awq_b200 import synth
    w1, w2 = synth.moe_layer_tensors(e, h, i, 128, seed=t + e)
    w1 = tuple(a.cuda() for a in w1)
    w2 = tuple(a.cuda() for a in w2)
    x = synth.activations(t, h, seed=t).cuda()
    logits = synth.gating_logits(t, e, seed=e).cuda()
    w, ids, _ = A.fused_topk(x, logits, k, True)
    d1, d2 = A.awq_repack(w1[0]), A.awq_repack(w2[0])
    assert d1.shape == w1[0].shape and d2.shape == w2[0].shape
    y0 = A.fused_experts(x, w1, w2, w, ids)
    y1 = A.fused_experts(x, w1, w2, w, ids, w1_decode=d1, w2_decode=d2)
    torch.cuda.synchronize()
    assert torch.equal(y0, y1)
    ref = O.fused_experts_fp32(x.cpu().numpy(), *[a.cpu().numpy() for a in w1],
                          *[a.cpu().numpy() for a in w2], w.cpu().numpy(), ids.cpu().numpy(), 128)
    assert O.rel_err(y1.cpu().numpy(), ref) < TOL
    with pytest.raises(ValueError):
        A.fused_experts(x, w1, w2, w, ids, w1_decode=d1)

    from awq_b200 import _lib
    lib = _lib.load()
    block = lib.awq_b200_moe_block_size(t, k, e, h, i, 128)
    sorted_ids, expert_ids, post = A.moe_align_block_size(ids, block, e, None)
    rows = -(-sorted_ids.numel() // block) * block

    def experts(q1, q2, flags, tables, capacity, nbytes):
        out = torch.full_like(x, float("nan"))
        scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        rc = lib.awq_b200_moe_experts(
            x.data_ptr(), q1.data_ptr(), w1[1].data_ptr(), w1[2].data_ptr(), q2.data_ptr(), w2[1].data_ptr(),
            w2[2].data_ptr(), w.data_ptr(), *tables, out.data_ptr(), t, k, e, h, i, 128, block, flags,
            capacity, scratch.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return rc, out

    tables = (sorted_ids.data_ptr(), expert_ids.data_ptr(), post.data_ptr())
    if block == 128:
        full = lib.awq_b200_moe_workspace_bytes(t, k, e, h, i)
        assert experts(d1, d2, 2, tables, sorted_ids.numel(), full)[0] == -2     # AWQ_B200_ERR_SHAPE
        return
    # activations of the permuted rows, rows by pair; the counters of the direct mode
    layout = lambda rows: -(-rows * i * 2 // 256) * 256 + -(-t * k * h * 2 // 256) * 256   # noqa: E731
    calls = [(0, tables, sorted_ids.numel(), layout(rows))]
    if block == 8 and t * k <= 64:
        calls.append((4, (None, ids.data_ptr(), None), t * k * 8, layout(t * k * 8) + 4096))
    for flags, table, capacity, nbytes in calls:
        rc, plain = experts(w1[0], w2[0], flags, table, capacity, nbytes)
        assert rc == 0
        rc, copies = experts(d1, d2, flags | 2, table, capacity, nbytes)
        assert rc == 0
        assert torch.equal(plain, copies)
        assert O.rel_err(copies.float().cpu().numpy(), ref) < TOL


# Batches of different sizes in turn, larger ones of NaN: nothing that an earlier call left in the
# scratch or in the routing tables may reach a result, however early the kernels of a call start.
@pytest.mark.parametrize("e,h,i,t,k", [(64, 1024, 256, 700, 4), (64, 1024, 256, 100, 4), (16, 512, 256, 2, 2)])
def test_batches_in_turn_do_not_see_each_other(A, e, h, i, t, k):
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=t)
    w1d, w2d = tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2)
    xd, nan = x.cuda(), torch.full((3 * t, h), float("nan"), dtype=torch.float16, device="cuda")
    weights, ids, _ = A.fused_topk(xd, logits.cuda(), k, True)
    other = [a.repeat(3, 1).flip(0).contiguous() for a in (weights, ids)]
    first = A.fused_experts(xd, w1d, w2d, weights, ids).clone()
    for _ in range(30):
        A.fused_experts(nan, w1d, w2d, *other)
        assert torch.equal(A.fused_experts(xd, w1d, w2d, weights, ids), first)


def _ts_forms(call):
    """(rows, mode, group, clusters, tokens beside the sums) of every gemm_ts kernel that a call launches, or nothing
    where the profiler sees no kernels."""
    import re
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    found = [re.search(r"gemm_ts_kernel<([^>]*)>", event.key) for event in prof.key_averages()]
    args = [re.sub(r"\(\w+\)", "", m.group(1)).replace(" ", "").split(",") for m in found if m]
    return [tuple(int(v) if v.isdigit() else int(v == "true") for v in a) for a in args]


# Blocks of 8 rows, then without a permutation: flags in both GEMMs, in gate_up alone, in none; flags and tokens in down.
@pytest.mark.parametrize("t,k,e,h,i,gate,down", [
    (5, 2, 8, 384, 640, 0, 0), (2, 6, 16, 2048, 256, 0, 1), (64, 4, 32, 512, 1024, 1, 1), (3, 1, 16, 512, 1152, None, 0),
    (9, 1, 32, 1024, 256, None, 1)])
def test_partial_tiles_of_experts_with_flags_and_with_tokens(A, t, k, e, h, i, gate, down):
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=t)
    w1d, w2d, xd = tuple(a.cuda() for a in w1), tuple(a.cuda() for a in w2), x.cuda()
    w, ids, _ = A.fused_topk(xd, logits.cuda(), k, True)
    want = A.fused_experts(xd, w1d, w2d, w, ids)
    forms = {f[1]: f for f in _ts_forms(lambda: A.fused_experts(xd, w1d, w2d, w, ids))}
    if forms:
        assert gate is None or forms[1][3:] == (0, gate)  # None: on clusters or not
        assert forms[2][3:] == (0, down)
    ref = O.fused_experts_fp32(x.numpy(), *[a.numpy() for a in w1], *[a.numpy() for a in w2], w.cpu().numpy(),
                               ids.cpu().numpy())
    assert O.rel_err(want.cpu().numpy(), ref) < TOL
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        out = [A.fused_experts(xd, w1d, w2d, w, ids) for _ in range(3)]
    for _ in range(20):
        for y in out:
            y.fill_(float("nan"))
        graph.replay()
        assert all(torch.equal(y, want) for y in out)
    torch.cuda.synchronize()


def test_partial_tiles_of_experts_with_any_scratch_and_replays(A):
    """Flags in gate_up, a token beside the sums in down: scratch full of other data, one buffer again and again, and
    replays of one graph whose tokens are the same every time."""
    from awq_b200 import _lib, ops
    t, k, e, h, i = 24, 4, 16, 2048, 768
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=5)
    w1d, w2d = (tuple(a.cuda() for a in ws) for ws in (w1, w2))
    xd = x.cuda()
    w, ids, _ = A.fused_topk(xd, logits.cuda(), k, True)
    block = _lib.load().awq_b200_moe_block_size(t, k, e, h, i, 128)
    assert block == 8
    want = A.fused_experts(xd, w1d, w2d, w, ids)
    sid, eid, npp = ops.moe_align_block_size(ids, block, e)
    need = _lib.load().awq_b200_moe_workspace_bytes(t, k, e, h, i)
    out = torch.empty_like(want)
    gen = torch.Generator(device="cuda").manual_seed(3)

    def call(scratch):
        rc = _lib.load().awq_b200_moe_experts(
            xd.data_ptr(), *[v.data_ptr() for v in (*w1d, *w2d)], w.data_ptr(), sid.data_ptr(), eid.data_ptr(),
            npp.data_ptr(), out.data_ptr(), t, k, e, h, i, 128, block, 0, sid.numel(), scratch.data_ptr(),
            scratch.numel(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
    for n in range(12):
        scratch = torch.randint(0, 256, (need,), dtype=torch.uint8, device="cuda", generator=gen)
        for _ in range(4):
            out.fill_(float("nan"))
            call(scratch)
            assert torch.equal(out, want), n
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        call(scratch)
        call(scratch)
    for _ in range(10):
        out.fill_(float("nan"))
        graph.replay()
        assert torch.equal(out, want)
    torch.cuda.synchronize()


@pytest.mark.parametrize("t,k,e,h,i", [(300, 2, 8, 512, 256), (160, 2, 4, 2048, 128)])
def test_prefill_calls_back_to_back_read_their_own_routing(A, t, k, e, h, i):
    """The down GEMM reads the tile table ahead of its wait for gate_up: calls with other routing right behind one
    another, in one buffer, give the bits that they give alone."""
    from awq_b200 import _lib, ops
    w1, w2, x, logits = _moe_case(e, h, i, t, k, seed=7)
    w1d, w2d = (tuple(a.cuda() for a in ws) for ws in (w1, w2))
    xd = x.cuda()
    assert _lib.load().awq_b200_moe_block_size(t, k, e, h, i, 128) == 128
    # most tokens on one expert, on another one, and spread out
    skews = [(0, 8.0), (e - 1, 8.0), (0, 0.0)]
    routed, want = [], []
    for expert, by in skews:
        ld = logits.cuda().clone()
        ld[:, expert] += by
        w, ids, _ = A.fused_topk(xd, ld, k, True)
        routed.append((w, *ops.moe_align_block_size(ids, 128, e)))
        want.append(A.fused_experts(xd, w1d, w2d, w, ids))
        torch.cuda.synchronize()
    need = _lib.load().awq_b200_moe_workspace_bytes(t, k, e, h, i)
    scratch = torch.empty(need, dtype=torch.uint8, device="cuda")
    order = [0, 1, 2, 1, 0, 2, 2, 0, 1] * 2
    outs = [torch.empty_like(want[0]) for _ in order]

    def calls():
        for n, out in zip(order, outs):
            w, sid, eid, npp = routed[n]
            rc = _lib.load().awq_b200_moe_experts(
                xd.data_ptr(), *[v.data_ptr() for v in (*w1d, *w2d)], w.data_ptr(), sid.data_ptr(), eid.data_ptr(),
                npp.data_ptr(), out.data_ptr(), t, k, e, h, i, 128, 128, 0, sid.numel(), scratch.data_ptr(),
                scratch.numel(), torch.cuda.current_stream().cuda_stream)
            assert rc == 0
    calls()
    for n, out in zip(order, outs):
        assert torch.equal(out, want[n]), n
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        calls()
    for _ in range(5):
        for out in outs:
            out.fill_(float("nan"))
        graph.replay()
        for n, out in zip(order, outs):
            assert torch.equal(out, want[n]), n
    torch.cuda.synchronize()
