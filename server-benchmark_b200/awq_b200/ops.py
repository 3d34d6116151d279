"""Operator-level API: same names, argument order and meaning as the vLLM ops the
cloudrift-ai/server-benchmark harness exercises (paths are inside the ``vllm`` package):

  awq_gemm(input, qweight, scales, qzeros, split_k_iters)      _custom_ops.py:576-587
  awq_dequantize(qweight, scales, zeros, split_k_iters, thx, thy)   _custom_ops.py:542-556
  fused_topk(hidden_states, gating_output, topk, renormalize, ...)
                                        model_executor/layers/fused_moe/router/fused_topk_router.py:69-113
  moe_align_block_size(topk_ids, block_size, num_experts, expert_map, ...)
                                        model_executor/layers/fused_moe/moe_align_block_size.py:11-103
  fused_experts(hidden_states, w1, w2, topk_weights, topk_ids, ...)
                                        model_executor/layers/fused_moe/fused_moe.py:1587-1631

Every function launches hand-written sm_100a kernels through the C ABI on the current CUDA
stream; nothing here computes on the CPU and nothing synchronises.  The operators called once per
layer go through the native host path (csrc/host_ops.cpp: checks, allocation, scratch, launch),
the load-time ones through ctypes.
"""
from __future__ import annotations

import torch

from . import _lib

PACK_FACTOR = 8
MOE_DIRECT_MAX_PAIRS = 64     # pairs up to which fused_experts goes direct, with at least twice as
                              # many experts (the limit of the C ABI, AWQ_B200_MOE_DIRECT_MAX_PAIRS;
                              # experts of the Qwen3-30B-A3B layer: 17 / 20 / 29 / 42 us direct
                              # against 21 / 25 / 33 / 46 us through the permutation at 1 / 2 / 4 / 8
                              # tokens)


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _require(t: torch.Tensor, name: str, dtype, ndim: int | None = None) -> None:
    if not isinstance(t, torch.Tensor):
        raise TypeError(f"{name} must be a torch.Tensor")
    if not t.is_cuda:
        raise ValueError(f"{name} must live on a CUDA device (there is no CPU path)")
    if t.dtype != dtype:
        raise ValueError(f"{name} must be {dtype}, got {t.dtype}")
    if ndim is not None and t.dim() != ndim:
        raise ValueError(f"{name} must have {ndim} dimensions, got {t.dim()}")
    if not t.is_contiguous():
        raise ValueError(f"{name} must be contiguous")


def reserve_workspace(nbytes: int, device: torch.device | str | None = None) -> None:
    """Make the current stream's scratch buffer at least ``nbytes`` large (load-time call: the buffer
    otherwise grows when a call needs more).  ``moe_workspace_bytes`` gives the need of the fused-MoE
    layer for a token count; the dense kernels never need more than the default.  Calls captured into
    a CUDA graph do not use it: they take their scratch from the graph's memory pool, so that graphs
    captured on one stream may be replayed on several at a time."""
    dev = torch.device(device) if device is not None else torch.device("cuda",
                                                                      torch.cuda.current_device())
    if nbytes > 0:
        index = dev.index if dev.index is not None else torch.cuda.current_device()
        _lib.native().workspace(index, int(nbytes))


def moe_workspace_bytes(tokens: int, topk: int, num_experts: int, hidden: int,
                        intermediate: int) -> int:
    """Scratch bytes ``fused_experts`` needs for up to ``tokens`` tokens (num_experts: the global
    expert count the routing is done over)."""
    return int(_lib.load().awq_b200_moe_workspace_bytes(tokens, topk, num_experts, hidden,
                                                        intermediate))


def awq_dequantize(qweight: torch.Tensor, scales: torch.Tensor, zeros: torch.Tensor,
                   split_k_iters: int = 0, thx: int = 0, thy: int = 0) -> torch.Tensor:
    """W fp16 [K, N] = (q - z) * s.  ``split_k_iters``, ``thx``, ``thy`` are accepted for
    signature compatibility (callers pass 0, 0, 0: quantization/awq.py:280) and ignored."""
    return _lib.native().dequantize(qweight, scales, zeros)


def awq_gemm(input: torch.Tensor, qweight: torch.Tensor, scales: torch.Tensor,
             qzeros: torch.Tensor, split_k_iters: int = 8, *, bias: torch.Tensor | None = None,
             kernel: int = _lib.KERNEL_AUTO, out: torch.Tensor | None = None) -> torch.Tensor:
    """y fp16 [M, N] = input [M, K] @ dequant(qweight), fp32 accumulation.

    ``split_k_iters`` is accepted and ignored (the split along K is chosen from the shape and
    the SM count).  ``bias``, ``kernel`` and ``out`` (a contiguous fp16 [M, N] tensor to write
    into, e.g. a view of a peer-mapped buffer) are keyword-only extensions.
    """
    return _lib.native().gemm(input, qweight, scales, qzeros, bias, kernel, out)


def awq_repack(qweight: torch.Tensor) -> torch.Tensor:
    """Decode-layout copy of ``qweight`` for ``awq_gemm(..., kernel=KERNEL_STREAM_RP)``.

    The copy holds, for every four rows k..k+3 and packed word column c, the four 32-bit
    words the streaming kernel otherwise builds with byte permutes: the low and the high
    halfwords of the row pairs (k, k+1) and (k+2, k+3).  It is returned with the shape of
    ``qweight`` ([K, N/8] int32; memory order [K/4, N/8, 4]) so that it can be passed where
    ``qweight`` goes; no other kernel understands it.  A stacked expert tensor [E, K, N/8] is
    repacked expert by expert (for ``fused_experts(..., w1_decode=, w2_decode=)``).  Load-time counterpart of the Marlin
    repack in vllm/model_executor/layers/quantization/awq_marlin.py:491-499.
    """
    _require(qweight, "qweight", torch.int32)
    if qweight.dim() not in (2, 3):
        raise ValueError("qweight must be [K, N/8] or stacked [E, K, N/8]")
    k, words = qweight.shape[-2:]
    if k % 4:
        raise ValueError("K must be a multiple of 4")
    out = torch.empty_like(qweight)
    if qweight.numel():
        # stacked experts: K % 4 == 0, so no row quad crosses an expert and the stack repacks
        # as one [E * K, N/8] matrix
        rc = _lib.load().awq_b200_repack_qweight(qweight.data_ptr(), out.data_ptr(),
                                                 qweight.numel() // words, words * 8, _stream())
        _lib.check("awq_b200_repack_qweight", rc)
        # Load-time operation: finish it here.  The GEMM kernels prefetch weights before they
        # wait for the kernel ahead of them in the stream, so a copy still being written must
        # not be handed to them.
        torch.cuda.current_stream().synchronize()
    return out


def awq_repack_kmajor(qweight: torch.Tensor) -> torch.Tensor:
    """K-major copy of ``qweight`` for ``awq_gemm(..., kernel=KERNEL_Q8)`` (up to 32 tokens).

    The same nibbles running along K, in 16 KB tiles of 256 output columns x one quantisation
    group, column slabs outermost (include/awq_b200.h, awq_b200_repack_kmajor).  Returned as
    int32 [K, ceil(N / 256) * 256 / 8]: the size of ``qweight`` when N is a multiple of 256.
    K must be a multiple of 128.  Load-time counterpart of the Marlin repack in
    vllm/model_executor/layers/quantization/awq_marlin.py:491-499.
    """
    _require(qweight, "qweight", torch.int32, 2)
    k, words = qweight.shape
    n = words * PACK_FACTOR
    lib = _lib.load()
    nbytes = int(lib.awq_b200_repack_kmajor_bytes(k, n))
    if nbytes == 0:
        raise ValueError("K must be a positive multiple of 128")
    out = torch.empty((k, nbytes // (4 * k)), dtype=torch.int32, device=qweight.device)
    rc = lib.awq_b200_repack_kmajor(qweight.data_ptr(), out.data_ptr(), k, n, _stream())
    _lib.check("awq_b200_repack_kmajor", rc)
    # load-time operation: the GEMM kernels prefetch weights before they wait for the kernel
    # ahead of them in the stream, so the copy must be complete before it is handed to them
    torch.cuda.current_stream().synchronize()
    return out


def wna16_to_awq(w: torch.Tensor, scales: torch.Tensor, zeros: torch.Tensor,
                 group_size: int = 128):
    """Stacked expert tensors in the byte layout of vLLM's MoE WNA16 method (w uint8 [E, N, K/2],
    scales fp16 [E, N, K/G], zeros uint8 [E, N/2, K/G]; moe_wna16.py:252-324) -> the AWQ
    checkpoint layout ``fused_experts`` takes: (qweight i32 [E, K, N/8], scales f16 [E, K/G, N],
    qzeros i32 [E, K/G, N/8]).  Load time; bit-exact inverse of vLLM's converter
    (moe_wna16.py:389-425)."""
    _require(w, "w", torch.uint8, 3)
    _require(scales, "scales", torch.float16, 3)
    _require(zeros, "zeros", torch.uint8, 3)
    e, n, half = w.shape
    k = 2 * half
    if n % PACK_FACTOR != 0 or k % group_size != 0:
        raise ValueError("N must be a multiple of 8 and K a multiple of the group size")
    g = k // group_size
    if scales.shape != (e, n, g) or zeros.shape != (e, n // 2, g):
        raise ValueError("scales / zeros shapes do not match w and the group size")
    qweight = torch.empty((e, k, n // PACK_FACTOR), dtype=torch.int32, device=w.device)
    qzeros = torch.empty((e, g, n // PACK_FACTOR), dtype=torch.int32, device=w.device)
    s_out = torch.empty((e, g, n), dtype=torch.float16, device=w.device)
    rc = _lib.load().awq_b200_wna16_to_awq(w.data_ptr(), scales.data_ptr(), zeros.data_ptr(),
                                           qweight.data_ptr(), s_out.data_ptr(),
                                           qzeros.data_ptr(), e, n, k, group_size, _stream())
    _lib.check("awq_b200_wna16_to_awq", rc)
    return qweight, s_out, qzeros


# ------------------------------------------------------------------------------- MoE


def fused_topk(hidden_states: torch.Tensor, gating_output: torch.Tensor, topk: int,
               renormalize: bool, indices_type: torch.dtype | None = None,
               scoring_func: str = "softmax"):
    """softmax -> top-k -> optional renormalise.  Returns (topk_weights f32 [T,k],
    topk_ids i32 [T,k], token_expert_indices i32 [T,k])."""
    if scoring_func != "softmax":
        raise ValueError(f"Unsupported scoring function: {scoring_func}")
    if indices_type not in (None, torch.int32):
        raise ValueError("indices_type must be torch.int32")
    return _lib.native().topk(hidden_states, gating_output, topk, renormalize)


def moe_align_block_size(topk_ids: torch.Tensor, block_size: int, num_experts: int,
                         expert_map: torch.Tensor | None = None, pad_sorted_ids: bool = False,
                         ignore_invalid_experts: bool = False):
    """Token -> expert permutation.  Returns (sorted_token_ids, expert_ids,
    num_tokens_post_padded), all int32 on the device."""
    _require(topk_ids, "topk_ids", torch.int32, 2)
    lib = _lib.load()
    t, k = topk_ids.shape
    cap = int(lib.awq_b200_moe_sorted_capacity(t * k, num_experts, block_size))
    if pad_sorted_ids:
        cap = -(-cap // block_size) * block_size
    dev = topk_ids.device
    sorted_ids = torch.empty((cap,), dtype=torch.int32, device=dev)
    nblk = -(-cap // block_size) if cap > 0 else 0
    expert_ids = torch.empty((nblk,), dtype=torch.int32, device=dev)
    num_post = torch.empty((1,), dtype=torch.int32, device=dev)
    emap = None
    if expert_map is not None and ignore_invalid_experts:
        _require(expert_map, "expert_map", torch.int32, 1)
        emap = expert_map
    rc = lib.awq_b200_moe_align_block_size(topk_ids.data_ptr(), t, k, num_experts, block_size,
                                           emap.data_ptr() if emap is not None else None,
                                           sorted_ids.data_ptr(), cap, expert_ids.data_ptr(),
                                           num_post.data_ptr(), _stream())
    _lib.check("awq_b200_moe_align_block_size", rc)
    if expert_map is not None and not ignore_invalid_experts:
        # same post-processing as the reference wrapper (moe_align_block_size.py:100-101);
        # unused trailing blocks stay -1
        used = expert_ids >= 0
        expert_ids = torch.where(used, expert_map[expert_ids.clamp(min=0).long()].to(torch.int32),
                                 expert_ids)
    return sorted_ids, expert_ids, num_post


def fused_experts(hidden_states: torch.Tensor, w1, w2, topk_weights: torch.Tensor,
                  topk_ids: torch.Tensor, inplace: bool = False, activation: str = "silu",
                  apply_router_weight_on_input: bool = False, global_num_experts: int = -1,
                  expert_map: torch.Tensor | None = None, group_size: int = 128,
                  w1_decode: torch.Tensor | None = None,
                  w2_decode: torch.Tensor | None = None, quant_config=None) -> torch.Tensor:
    """AWQ fused-MoE experts.  ``w1`` and ``w2`` are (qweight, scales, qzeros) triples of the
    stacked AWQ tensors: w1 = (i32 [E,H,2I/8], f16 [E,H/G,2I], i32 [E,H/G,2I/8]),
    w2 = (i32 [E,I,H/8], f16 [E,I/G,H], i32 [E,I/G,H/8]).  Returns fp16 [T, H].

    The form of vLLM's ``fused_experts`` (fused_moe/fused_moe.py:1587-1599) is accepted too:
    ``w1`` / ``w2`` the two stacked qweight tensors and ``quant_config`` an object carrying
    ``w1_scale``, ``w2_scale``, ``w1_zp``, ``w2_zp`` (a ``FusedMoEQuantConfig``, e.g. from
    ``int4_w4a16_moe_quant_config``); its ``block_shape[1]``, when set, is the group size.

    ``w1_decode`` / ``w2_decode`` (both or neither): ``awq_repack`` of the two stacked qweights.
    Accepted and checked; the expert kernels read ``w1`` / ``w2``, for which the checkpoint layout is
    the faster one."""
    if activation != "silu":
        raise ValueError("only the silu activation is implemented")
    if apply_router_weight_on_input:
        raise ValueError("apply_router_weight_on_input is not implemented")
    if quant_config is not None:
        if not (torch.is_tensor(w1) and torch.is_tensor(w2)):
            raise ValueError("with quant_config, w1 and w2 are the stacked qweight tensors")
        w1 = (w1, quant_config.w1_scale, quant_config.w1_zp)
        w2 = (w2, quant_config.w2_scale, quant_config.w2_zp)
        if w1[1] is None or w1[2] is None or w2[1] is None or w2[2] is None:
            raise ValueError("quant_config must carry w1_scale, w2_scale, w1_zp and w2_zp")
        shape = getattr(quant_config, "block_shape", None)
        if shape is not None and len(shape) == 2 and shape[1]:
            group_size = int(shape[1])
    elif torch.is_tensor(w1) or torch.is_tensor(w2):
        raise ValueError("w1 and w2 are (qweight, scales, qzeros) triples, or tensors together "
                         "with quant_config")
    return _lib.native().experts(hidden_states, tuple(w1), tuple(w2), topk_weights, topk_ids,
                                 inplace, global_num_experts, expert_map, group_size, w1_decode,
                                 w2_decode, MOE_DIRECT_MAX_PAIRS)


def fused_moe(hidden_states: torch.Tensor, w1, w2, gating_output: torch.Tensor, topk: int,
              renormalize: bool, inplace: bool = False, group_size: int = 128) -> torch.Tensor:
    """Routing followed by the experts: fused_topk then fused_experts (the historical
    ``fused_moe`` entry point older call sites use)."""
    w, ids, _ = fused_topk(hidden_states, gating_output, topk, renormalize)
    return fused_experts(hidden_states, w1, w2, w, ids, inplace=inplace, group_size=group_size)
