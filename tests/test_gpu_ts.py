"""Parity of the decode-size tcgen05 kernel (weights registers -> TMEM, A operand in TMEM) with
the CPU oracle, through the C ABI."""
import ctypes

import numpy as np
import pytest
import torch

from cuts import cut
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


def run_case(A, kernel, m, k, n, seed=0, bias=False):
    from awq_b200 import synth
    qw, s, qz = synth.awq_linear_tensors(k, n, 128, seed=seed)
    x = synth.activations(m, k, seed=seed + 1)
    b = torch.randn(n, generator=torch.Generator().manual_seed(seed)).half() if bias else None
    y = A.awq_gemm(x.cuda(), qw.cuda(), s.cuda(), qz.cuda(), 8,
                   bias=b.cuda() if bias else None, kernel=kernel)
    torch.cuda.synchronize()
    assert device_status() == 0, "a bounded wait ran out"
    ref = O.awq_gemm_fp32(x.numpy(), qw.numpy(), s.numpy(), qz.numpy(), 128)
    if bias:
        ref = ref + b.numpy().astype(np.float32)
    y = y.cpu().numpy()
    assert np.isfinite(y.astype(np.float32)).all()
    err = O.rel_err(y, ref)
    assert err < TOL, f"rel err {err}"
    assert O.elementwise_ok(y, ref, TOL)


SHAPES = [
    (16, 128, 256),     # one stage, one slab
    (16, 256, 256),     # two stages
    (16, 1024, 512),    # ring wraps, two slabs
    (1, 512, 256), (3, 384, 32), (9, 640, 288),   # ragged M, N edge inside a slab
    (16, 8192, 8192), (4, 3712, 8192), (16, 2048, 1536),
]


@pytest.mark.parametrize("m,k,n", SHAPES)
def test_ts_exact_vs_oracle(A, m, k, n):
    run_case(A, A.KERNEL_TS_EXACT, m, k, n, seed=m + n)


@pytest.mark.parametrize("m,k,n", SHAPES)
def test_ts_fast_vs_oracle(A, m, k, n):
    run_case(A, A.KERNEL_TS, m, k, n, seed=m + k)


def test_ts_bias_determinism_and_agreement_with_stream_kernel(A):
    from awq_b200 import synth
    run_case(A, A.KERNEL_TS, 16, 2048, 768, seed=4, bias=True)
    m, k, n = 16, 4096, 2048
    qw, s, qz = [a.cuda() for a in synth.awq_linear_tensors(k, n, 128, seed=8)]
    x = synth.activations(m, k, seed=9).cuda()
    y1 = A.awq_gemm(x, qw, s, qz, 8, kernel=A.KERNEL_TS)
    y2 = A.awq_gemm(x, qw, s, qz, 8, kernel=A.KERNEL_TS)
    assert torch.equal(y1, y2)
    y3 = A.awq_gemm(x, qw, s, qz, 8, kernel=A.KERNEL_STREAM)
    assert O.rel_err(y1.cpu().numpy(), y3.float().cpu().numpy()) < 2e-3
    assert device_status() == 0


# Sizes at which the work split and the token variants change: fewer units than CTAs, slabs shared by
# several CTAs, ranges that end on a slab, whole slabs only, N edge inside a slab, every token variant
# at its ends.  Units of a CTA's range (0: whole slabs): asserted, as the cut follows from a cost.
RANGES = {(1, 128, 32): 0, (4, 8192, 1280): 4, (5, 384, 4768): 0, (8, 2432, 8192): 5, (12, 1024, 38144): 9,
          (16, 29568, 288): 15, (9, 3712, 2592): 5, (13, 4096, 1056): 4}


@pytest.mark.parametrize("m,k,n", list(RANGES))
def test_ts_work_split_edges(A, m, k, n):
    assert cut(m, k, n, 128, A.KERNEL_TS)[1:4] == (next(t for t in (4, 8, 16) if m <= t), RANGES[m, k, n], 0)
    run_case(A, A.KERNEL_TS, m, k, n, seed=m + n, bias=m % 2 == 1)

    # replays of one captured launch interleaved with another shape on the same scratch, and a call
    # without scratch (whole slabs)
    from awq_b200 import _lib, synth
    qw, s, qz = [a.cuda() for a in synth.awq_linear_tensors(k, n, 128, seed=1)]
    x = synth.activations(m, k, seed=2).cuda()
    y = A.awq_gemm(x, qw, s, qz, 8, kernel=A.KERNEL_TS)
    out = torch.empty_like(y)
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        A.awq_gemm(x, qw, s, qz, 8, kernel=A.KERNEL_TS, out=out)
        stream.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            A.awq_gemm(x, qw, s, qz, 8, kernel=A.KERNEL_TS, out=out)
        for _ in range(3):
            out.zero_()
            graph.replay()
            A.awq_gemm(x[:1].contiguous(), qw, s, qz, 8, kernel=A.KERNEL_TS)
            assert torch.equal(out, y)
    torch.cuda.synchronize()
    rc = _lib.load().awq_b200_gemm(x.data_ptr(), qw.data_ptr(), s.data_ptr(), qz.data_ptr(), None,
                                   out.data_ptr(), m, n, k, 128, A.KERNEL_TS, None, 0,
                                   torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    # the same products, summed in one piece: fp32 rounding and one fp16 rounding apart
    assert O.rel_err(out.cpu().numpy(), y.float().cpu().numpy()) < 2e-3
    assert device_status() == 0


# Two quantisation groups of 64 in a unit: one unit in all, shared and whole slabs, the token counts of
# every variant at their edges, a slab past N, bias.
RANGES_64 = {(1, 128, 32): 0, (4, 8192, 1280): 4, (5, 384, 2080): 0, (8, 4096, 4768): 5, (9, 15360, 544): 8,
             (16, 1536, 28704): 0}


@pytest.mark.parametrize("m,k,n", list(RANGES_64))
@pytest.mark.parametrize("bias", [False, True])
def test_ts_groups_of_64(A, m, k, n, bias):
    from awq_b200 import synth
    assert cut(m, k, n, 64, A.KERNEL_TS)[2:4] == (RANGES_64[m, k, n], 0)
    qw, s, qz = synth.awq_linear_tensors(k, n, 64, seed=m + n)
    x = synth.activations(m, k, seed=k)
    b = synth.activations(1, n, seed=3)[0] if bias else None
    ref = O.awq_gemm_fp32_torch(x, qw, s, qz, 64).numpy() + (b.float().numpy() if bias else 0)
    y = [A.awq_gemm(x.cuda(), qw.cuda(), s.cuda(), qz.cuda(), 8, kernel=A.KERNEL_TS,
                    bias=b.cuda() if bias else None) for _ in range(2)]
    torch.cuda.synchronize()
    assert device_status() == 0, "a bounded wait ran out"
    assert torch.equal(y[0], y[1])
    # fp32 sums of exact products; the output's 2^-11 is far inside TOL
    assert O.rel_err(y[0].cpu().numpy(), ref) < TOL


@pytest.mark.parametrize("kernel,m,k,n", [("KERNEL_TS", 5, 8192, 1280), ("KERNEL_WT", 40, 8192, 1312),
                                          ("KERNEL_TS", 3, 8192, 1280), ("KERNEL_TS", 14, 8192, 1280),
                                          ("KERNEL_AUTO", 12, 1024, 38144), ("KERNEL_AUTO", 20, 2048, 38144)])
def test_scratch_may_be_any_buffer_with_any_content(A, kernel, m, k, n):
    """Shared slabs and tiles with more scratch buffers, one after the other, than a table of them could hold,
    each full of other data, and one buffer again and again: always the same bits."""
    from awq_b200 import _lib, synth
    qw, s, qz = (t.cuda() for t in synth.awq_linear_tensors(k, n, 128, seed=1))
    x = synth.activations(m, k, seed=2).cuda()
    lib, kernel = _lib.load(), getattr(A, kernel)
    assert cut(m, k, n, 128, kernel).chunk > 0  # handed over through the scratch
    need = lib.awq_b200_gemm_workspace_bytes(m, n, k, 128, kernel)
    assert need > 0
    step = -(-need // 256) * 256
    pool = torch.randint(0, 256, (150 * step,), dtype=torch.uint8, device="cuda",
                         generator=torch.Generator(device="cuda").manual_seed(3))
    pool[:step] = 255
    pool[step:2 * step] = 0
    outs = torch.full((300, m, n), float("nan"), dtype=torch.float16, device="cuda")
    for i in range(300):
        scratch = pool[min(i, 149) * step:]
        rc = lib.awq_b200_gemm(x.data_ptr(), qw.data_ptr(), s.data_ptr(), qz.data_ptr(), None,
                               outs[i].data_ptr(), m, n, k, 128, kernel, scratch.data_ptr(), step,
                               torch.cuda.current_stream().cuda_stream)
        assert rc == 0
    torch.cuda.synchronize()
    assert device_status() == 0, "a bounded wait ran out"
    assert torch.isfinite(outs[0].float()).all()
    assert all(torch.equal(outs[0], y) for y in outs[1:])


@pytest.mark.parametrize("m,group", [(5, 128), (20, 64)])
def test_automatic_choice_without_enough_scratch_takes_the_streaming_kernel(A, m, group):
    """Scratch that is too small or misaligned serves no hand-over: the call runs as without any."""
    from awq_b200 import _lib, synth
    k, n = 8192, 1280
    dev = [t.cuda() for t in (synth.activations(m, k, seed=2), *synth.awq_linear_tensors(k, n, group, seed=1))]
    lib = _lib.load()
    need = lib.awq_b200_gemm_workspace_bytes(m, n, k, group, 0)
    pool = torch.empty(need + 512, dtype=torch.uint8, device="cuda")
    want = A.awq_gemm(*dev, 8, kernel=A.KERNEL_STREAM)
    for ptr, size in ((None, 0), (pool.data_ptr(), need - 1), (pool.data_ptr() + 16, need)):
        y = torch.empty_like(want)
        rc = lib.awq_b200_gemm(*[t.data_ptr() for t in dev], None, y.data_ptr(), m, n, k, group, 0, ptr, size,
                               torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        assert torch.equal(y, want)


def _layers(A, m):
    """A linear as the automatic choice cuts it (clusters), one that is handed over through the scratch, a MoE layer."""
    from awq_b200 import synth
    ranges = A.KERNEL_TS if m <= 16 else A.KERNEL_WT
    assert cut(m, 8192, 1280, 128).cluster > 0 and cut(m, 8192, 1280, 128, ranges).chunk > 0
    dense = [t.cuda() for t in (synth.activations(m, 8192, seed=m), *synth.awq_linear_tensors(8192, 1280, 128, seed=1))]
    e, h, i, k = 16, 1024, 256, 4
    w1, w2 = (tuple(t.cuda() for t in w) for w in synth.moe_layer_tensors(e, h, i, 128, seed=2))
    x, logits = synth.activations(m, h, seed=m).cuda(), synth.gating_logits(m, e, seed=m).cuda()
    return lambda: (A.awq_gemm(*dense, 8), A.awq_gemm(*dense, 8, kernel=ranges), A.fused_moe(x, w1, w2, logits, k, True))


def test_graphs_captured_on_one_stream_run_side_by_side(A):
    """Two captured steps with shared slabs and tiles, from one capture stream, replayed on two streams at
    a time: each has scratch of its own."""
    steps = [_layers(A, 5), _layers(A, 40)]
    want = [[y.clone() for y in step()] for step in steps]
    torch.cuda.synchronize()
    graphs, outs = [], []
    for step in steps:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):       # the default capture stream, the same for both
            outs.append(step())
        graphs.append(graph)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(20):
        for graph, stream in zip(graphs, streams):
            with torch.cuda.stream(stream):
                for _ in range(10):
                    graph.replay()
        torch.cuda.synchronize()
        for ys, refs in zip(outs, want):
            assert all(torch.equal(y, ref) for y, ref in zip(ys, refs))
    assert device_status() == 0, "a bounded wait ran out"


def test_capture_on_a_new_stream_takes_calls_of_any_size(A):
    """A stream's first captured calls: a linear, then a fused-MoE layer with a larger need."""
    from awq_b200 import synth
    small = _layers(A, 5)
    e, h, i, k, t = 16, 2048, 768, 8, 1024
    w1, w2 = (tuple(a.cuda() for a in w) for w in synth.moe_layer_tensors(e, h, i, 128, seed=2))
    x, logits = synth.activations(t, h, seed=t).cuda(), synth.gating_logits(t, e, seed=t).cuda()
    want = A.fused_moe(x, w1, w2, logits, k, True)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        small()
        y = A.fused_moe(x, w1, w2, logits, k, True)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)


# Slabs shared by clusters of 2, 3, 4, 5, 6, 8 and 16 CTAs, units that do not divide by them, one unit a CTA, an edge of N
# inside a slab, the token variants at their ends; ranges over the whole GPU with 17 to 32 tokens, whole slabs, one unit in
# all.  CTAs of a cluster on a B200, or units of a range: which of the two is asserted on the GPU, which number on the CPU.
CLUSTERS = {
    (1, 1024, 8192, 128): (2, 0), (30, 1024, 8192, 64): (2, 0), (3, 2176, 5120, 128): (3, 0),
    (32, 2176, 5152, 128): (3, 0), (17, 4096, 4064, 64): (4, 0), (9, 640, 1312, 128): (5, 0),
    (25, 12288, 6176, 128): (5, 0), (24, 8192, 5120, 64): (6, 0), (12, 2048, 1024, 64): (8, 0),
    (16, 8192, 1280, 128): (16, 0), (31, 8192, 1280, 128): (16, 0), (4, 16384, 992, 64): (16, 0),
    (5, 256, 256, 128): (0, 0), (20, 128, 32, 128): (0, 0), (23, 8192, 38176, 128): (0, 65),
    (18, 4096, 28704, 64): (0, 0), (20, 256, 2080, 128): (0, 0), (20, 512, 1056, 128): (4, 0), (2, 512, 1056, 128): (4, 0),
    (7, 768, 544, 128): (6, 0), (27, 4096, 20512, 64): (0, 18), (32, 2048, 38144, 128): (0, 17)}


@pytest.mark.parametrize("m,k,n,group", list(CLUSTERS))
@pytest.mark.parametrize("bias", [False, True])
def test_ts_clusters_and_up_to_32_tokens(A, m, k, n, group, bias):
    """Nothing but the output is rounded to fp16, and the bits do not depend on timing."""
    from awq_b200 import synth
    got, (ctas, units) = cut(m, k, n, group), CLUSTERS[m, k, n, group]
    assert (got.kernel, got.cluster > 0, got.chunk > 0) == (A.KERNEL_TS, ctas > 0, units > 0)
    qw, s, qz = synth.awq_linear_tensors(k, n, group, seed=m + n)
    x = synth.activations(m, k, seed=k)
    b = synth.activations(1, n, seed=3)[0] if bias else None
    cols = torch.arange(n)[max(0, n - 1024):]  # of the oracle: the last ones, with the edge
    ref = x.double() @ torch.from_numpy(O.dequantize_fp32(
        qw[:, cols[0] // 8:].numpy(), s[:, cols].numpy(), qz[:, cols[0] // 8:].numpy(), group)).double()
    if bias:
        ref += b[cols].double()
    outs = [A.awq_gemm(x.cuda(), qw.cuda(), s.cuda(), qz.cuda(), 8, bias=b.cuda() if bias else None)
            for _ in range(3)]
    torch.cuda.synchronize()
    assert device_status() == 0, "a bounded wait ran out"
    assert all(torch.equal(outs[0], y) for y in outs[1:])
    error = (outs[0].cpu()[:, cols].double() - ref).norm()
    # 5 %: the fp32 sums, K * 2^-24 of their terms' size at most, move few values to the other side
    assert error < 1.05 * (ref.half().double() - ref).norm()


def test_explicit_ts_takes_16_rows_at_most(A):
    from awq_b200 import synth
    dev = [t.cuda() for t in (synth.activations(17, 256, seed=2), *synth.awq_linear_tensors(256, 256, 128, seed=1))]
    with pytest.raises(ValueError):
        A.awq_gemm(*dev, 8, kernel=A.KERNEL_TS)
