"""Parity of the weights-in-tensor-memory tcgen05 kernel (dequantised weights registers -> TMEM as
the A operand, activations as the B operand) with the CPU oracle, through the C ABI."""
import ctypes

import numpy as np
import pytest
import torch

import cuts
from oracle import awq_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-2


@pytest.fixture(scope="module")
def A(built_library):
    import awq_b200
    assert torch.cuda.is_available()
    return awq_b200


def device_status():
    from awq_b200 import _lib
    v = ctypes.c_int(-1)
    assert _lib.load().awq_b200_device_status(ctypes.byref(v)) == 0
    return v.value


def run_case(A, m, k, n, seed=0, bias=False):
    from awq_b200 import synth
    qw, s, qz = synth.awq_linear_tensors(k, n, 128, seed=seed)
    x = synth.activations(m, k, seed=seed + 1)
    b = torch.randn(n, generator=torch.Generator().manual_seed(seed)).half() if bias else None
    y = A.awq_gemm(x.cuda(), qw.cuda(), s.cuda(), qz.cuda(), 8,
                   bias=b.cuda() if bias else None, kernel=A.KERNEL_WT)
    torch.cuda.synchronize()
    assert device_status() == 0, "a bounded wait ran out"
    ref = O.awq_gemm_fp32_torch(x, qw, s, qz, 128).numpy()
    if bias:
        ref = ref + b.numpy().astype(np.float32)
    y = y.cpu().numpy()
    assert np.isfinite(y.astype(np.float32)).all()
    err = O.rel_err(y, ref)
    assert err < TOL, f"rel err {err}"
    assert O.elementwise_ok(y, ref, TOL)


SHAPES = [
    (64, 128, 256),      # one stage, one slab, 64-token tile
    (64, 256, 256),      # two stages: both A ring halves
    (48, 1024, 512),     # ring wraps, ragged M
    (128, 640, 288),     # 128-token tile, N edge inside a slab
    (100, 2048, 1536), (33, 384, 32), (1, 512, 256), (17, 3712, 8192),
    (256, 1024, 1024),   # two token tiles
    (300, 2048, 512),    # ragged last token tile
    (1024, 8192, 1024),
]


@pytest.mark.parametrize("m,k,n", SHAPES)
def test_wt_vs_oracle(A, m, k, n):
    run_case(A, m, k, n, seed=m + n)


def test_wt_bias_and_repeat(A):
    run_case(A, 64, 1024, 512, seed=5, bias=True)
    run_case(A, 200, 1024, 512, seed=6, bias=True)


def test_wt_deterministic(A):
    from awq_b200 import synth
    qw, s, qz = [a.cuda() for a in synth.awq_linear_tensors(4096, 2048, 128, seed=3)]
    x = synth.activations(96, 4096, seed=4).cuda()
    y0 = A.awq_gemm(x, qw, s, qz, 8, kernel=A.KERNEL_WT)
    for _ in range(3):
        assert torch.equal(y0, A.awq_gemm(x, qw, s, qz, 8, kernel=A.KERNEL_WT))


def test_wt_rejects_unsupported_shapes(A):
    from awq_b200 import synth
    qw, s, qz = [a.cuda() for a in synth.awq_linear_tensors(256, 264, 128, seed=1)]  # N % 32 != 0
    x = synth.activations(64, 256).cuda()
    with pytest.raises(ValueError):
        A.awq_gemm(x, qw, s, qz, 8, kernel=A.KERNEL_WT)


# Sizes at which the pair kernel's work split and tiles change: fewer tiles than pairs (a tile shared
# by two to five pairs), exactly one tile, a chunk that ends inside / on a tile, the second CTA of a
# pair past N, both group sizes, token counts around the tile (16, 128 / 144: one or two
# accumulators) and above one tile (ragged last one).
@pytest.mark.parametrize("m,k,n,group", [
    (17, 1024, 8192, 128), (24, 8192, 1280, 64), (33, 3712, 1568, 128), (16, 128, 32, 64),
    (127, 2048, 4768, 64), (128, 8192, 2048, 128), (129, 4096, 160, 128), (144, 1280, 19200, 128),
    (255, 2048, 8224, 64), (257, 384, 544, 128), (1000, 512, 2592, 64),
])
def test_wt_work_split_edges(A, m, k, n, group):
    from awq_b200 import synth
    qw, s, qz = synth.awq_linear_tensors(k, n, group, seed=m)
    x = synth.activations(m, k, seed=n)
    ref = O.awq_gemm_fp32_torch(x, qw, s, qz, group).numpy()
    dev = [a.cuda() for a in (qw, s, qz)]
    xd = x.cuda()
    y = A.awq_gemm(xd, *dev, 8, kernel=A.KERNEL_WT)
    torch.cuda.synchronize()
    assert device_status() == 0, "a bounded wait ran out"
    # fp16 weights and output: 2^-11 each, far inside TOL
    assert O.rel_err(y.cpu().numpy(), ref) < TOL
    assert O.elementwise_ok(y.cpu().numpy(), ref, TOL)

    # replays of one captured launch, interleaved with another shape on the same scratch
    out = torch.empty_like(y)
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        A.awq_gemm(xd, *dev, 8, kernel=A.KERNEL_WT, out=out)
        stream.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            A.awq_gemm(xd, *dev, 8, kernel=A.KERNEL_WT, out=out)
        for _ in range(3):
            out.zero_()
            graph.replay()
            A.awq_gemm(xd[:16].contiguous(), *dev, 8, kernel=A.KERNEL_WT)
            assert torch.equal(out, y)
    torch.cuda.synchronize()

    # without scratch whole tiles are distributed: the same sums, in one piece
    from awq_b200 import _lib
    rc = _lib.load().awq_b200_gemm(xd.data_ptr(), *[a.data_ptr() for a in dev], None, out.data_ptr(), m,
                                   n, k, group, A.KERNEL_WT, None, 0,
                                   torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    assert O.rel_err(out.cpu().numpy(), ref) < TOL


# Shared tiles collected from up to five pairs through the shared-memory ring: more pieces of 32 tokens
# than it has slots, a last piece of 16 tokens, several token tiles with a ragged last one, a slab past N.
@pytest.mark.parametrize("m,k,n,group", [
    (40, 8192, 1312, 128), (97, 16384, 64, 64), (239, 6400, 2560, 128), (333, 8192, 1280, 128),
    (700, 8192, 1280, 64),
])
def test_wt_collected_tiles(A, m, k, n, group):
    from awq_b200 import synth
    qw, s, qz = synth.awq_linear_tensors(k, n, group, seed=n)
    x = synth.activations(m, k, seed=m)
    ref = O.awq_gemm_fp32_torch(x, qw, s, qz, group).numpy()
    dev = [a.cuda() for a in (x, qw, s, qz)]
    y = [A.awq_gemm(*dev, 8, kernel=A.KERNEL_WT) for _ in range(3)]
    torch.cuda.synchronize()
    assert device_status() == 0, "a bounded wait ran out"
    assert torch.equal(y[0], y[1]) and torch.equal(y[0], y[2])
    # fp16 weights and output: 2^-11 each, far inside TOL
    assert O.rel_err(y[0].cpu().numpy(), ref) < TOL
    assert O.elementwise_ok(y[0].cpu().numpy(), ref, TOL)


# Tiles of more than 128 tokens, one accumulator.  Whole ones, whose epilogue goes through shared memory: every tile size
# from 144 to 256 (4 to 13 stages of packed words), one to nine units a tile, a last tile of few tokens, a slab past N,
# first several tiles to a pair, then one.  Last, split ones, whose epilogue does not.  (m, k, n, group, tokens of a tile,
# split): asserted, as the cut follows from a cost.
CUT_CASES = [
    (400, 640, 9504, 128, 144, False), (777, 384, 9504, 64, 160, False), (500, 128, 9504, 128, 176, False),
    (900, 640, 9504, 64, 192, False), (777, 256, 8224, 128, 208, False), (430, 1152, 9472, 128, 224, False),
    (900, 512, 8224, 64, 240, False), (1000, 640, 8224, 128, 256, False),
    (264, 1024, 8192, 128, 144, False), (150, 4096, 11040, 64, 160, False), (400, 1024, 8192, 128, 208, False),
    (511, 4096, 8192, 64, 256, False), (774, 8192, 544, 128, 144, True), (291, 7680, 3360, 64, 160, True),
]


def cut(m, k, n, group, cta_pairs):
    """(tokens of a tile, units of a pair's range or 0, epilogue through shared memory)"""
    from awq_b200 import _lib
    v = [ctypes.c_int(-1) for _ in range(3)]
    rc = _lib.load().awq_b200_gemm_wt_cut(m, n, k, group, cta_pairs, *[ctypes.byref(x) for x in v])
    assert rc == 0
    return tuple(x.value for x in v)


@pytest.mark.parametrize("m,k,n,group,tokens,split", CUT_CASES)
def test_wt_wide_tiles(A, m, k, n, group, tokens, split):
    got = cut(m, k, n, group, 0)
    assert (got[0], got[1] > 0, got[2]) == (tokens, split, 0 if split else 1)
    from awq_b200 import synth
    qw, s, qz = synth.awq_linear_tensors(k, n, group, seed=m)
    x = synth.activations(m, k, seed=n)
    b = torch.randn(n, generator=torch.Generator().manual_seed(k)).half()
    ref = O.awq_gemm_fp32_torch(x, qw, s, qz, group).numpy() + b.numpy().astype(np.float32)
    dev = [a.cuda() for a in (x, qw, s, qz)]
    y = [A.awq_gemm(*dev, 8, bias=b.cuda(), kernel=A.KERNEL_WT) for _ in range(3)]
    torch.cuda.synchronize()
    assert device_status() == 0, "a bounded wait ran out"
    assert torch.equal(y[0], y[1]) and torch.equal(y[0], y[2])
    # fp16 weights and output: 2^-11 each, far inside TOL
    assert O.rel_err(y[0].cpu().numpy(), ref) < TOL
    assert O.elementwise_ok(y[0].cpu().numpy(), ref, TOL)


# Tiles shared by clusters: two to eight pairs a tile, two tiles for three pairs, units that do not divide by the pairs, one
# unit a pair, an edge of N, several tiles of tokens with a shorter last one, one accumulator (tiles above 64
# tokens, and above 128); and, (0, 0), calls near them that are faster in ranges.  CTAs and tiles of a cluster on a B200:
# asserted on the CPU, on the GPU whether there are clusters.
CLUSTERS = {
    (40, 1024, 4096, 128): (4, 1), (130, 512, 2048, 64): (0, 0), (33, 384, 1056, 128): (6, 1),
    (97, 640, 2048, 128): (0, 0), (77, 4096, 4096, 64): (4, 1), (100, 8192, 1280, 128): (10, 1),
    (300, 8192, 1312, 64): (6, 1), (150, 11008, 1536, 128): (8, 1), (60, 16384, 544, 128): (16, 1),
    (100, 8192, 10240, 128): (6, 2), (48, 4352, 10208, 64): (6, 2), (250, 8192, 5120, 128): (6, 2),
    (500, 8192, 2080, 128): (0, 0), (48, 2304, 64, 128): (12, 1), (33, 640, 64, 128): (6, 1), (130, 2304, 2080, 128): (6, 1),
    (400, 4096, 2080, 64): (4, 1), (64, 1280, 2080, 128): (6, 2)}


@pytest.mark.parametrize("m,k,n,group", list(CLUSTERS))
@pytest.mark.parametrize("bias", [False, True])
def test_wt_clusters_share_tiles(A, m, k, n, group, bias):
    """Weights rounded to (q - z) * s and the output are all that is rounded to fp16; the bits do not depend on timing."""
    from awq_b200 import synth
    assert (cuts.cut(m, k, n, group).cluster > 0) == (CLUSTERS[m, k, n, group] != (0, 0))
    assert cuts.cut(m, k, n, group, A.KERNEL_WT).cluster == 0
    qw, s, qz = synth.awq_linear_tensors(k, n, group, seed=m + n)
    x = synth.activations(m, k, seed=k)
    b = synth.activations(1, n, seed=3)[0] if bias else None
    c = max(0, n - 768)  # first column of the oracle: the last ones, with the edge
    w = O.dequantize_fp32(qw[:, c // 8:].numpy(), s[:, c:].numpy(), qz[:, c // 8:].numpy(), group)
    ref = x.double() @ torch.from_numpy(w).half().double()  # the fp32 product of 5 and 11 bits is exact
    if bias:
        ref += b[c:].double()
    dev = [t.cuda() for t in (x, qw, s, qz)]
    outs = [A.awq_gemm(*dev, 8, bias=b.cuda() if bias else None) for _ in range(3)]
    named = A.awq_gemm(*dev, 8, bias=b.cuda() if bias else None, kernel=A.KERNEL_WT)
    torch.cuda.synchronize()
    assert device_status() == 0, "a bounded wait ran out"
    assert all(torch.equal(outs[0], y) for y in outs[1:])
    rounding = (ref.half().double() - ref).norm()
    # 5 %: the fp32 sums, K * 2^-24 of their terms' size at most, move few values to the other side
    for y in (outs[0], named):
        assert (y.cpu()[:, c:].double() - ref).norm() < 1.05 * rounding


# Ranges of 65 to 128 tokens on either side of the K from which they have one accumulator and six A slots, which is larger
# for 128 tokens in groups of 128 and ranges of more than a tile: a tile shared by pairs, three tiles in a range, tiles of
# 48, 80, 112 and 128 tokens, a slab past N.
ACCUMULATORS = {(100, 7168, 8224, 64): 1, (100, 7040, 8224, 128): 2, (72, 7168, 20512, 128): 1, (128, 7296, 1568, 128): 2,
                (128, 8192, 10784, 128): 1, (128, 7168, 20512, 128): 2, (128, 11264, 20512, 128): 1,
                (128, 7168, 20512, 64): 1}


@pytest.mark.parametrize("m,k,n,group", list(ACCUMULATORS))
def test_wt_ranges_with_one_or_two_accumulators(A, m, k, n, group):
    got = cuts.cut(m, k, n, group, A.KERNEL_WT)
    assert got.chunk > 0 and got.accumulators == ACCUMULATORS[m, k, n, group]
    test_wt_work_split_edges(A, m, k, n, group)
