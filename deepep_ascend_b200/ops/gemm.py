"""Python front end of the tcgen05 GEMM kernels (``csrc/kernels/gemm_sm100.cu``) and of the small MoE helpers.

No counterpart in the reference, which contains no tensor-core code; these kernels exist for the fused MoE layer
and for the all-gather / reduce-scatter fused GEMMs.
"""
from typing import Optional, Tuple

import torch

from .. import _native

BLOCK_M = 128   # rows of one output tile; expert segments of the grouped GEMM are aligned to it


def _core_of(buffer):
    return None if buffer is None else buffer.core


def gemm_nt(a: torch.Tensor, b: torch.Tensor, out: Optional[torch.Tensor] = None, num_sms: int = 0, buffer=None) -> torch.Tensor:
    """``a [M, K] @ b [N, K]^T -> bf16 [M, N]`` (bf16 operands, fp32 accumulation in tensor memory).  With ``buffer``
    (an ``ElasticBuffer``) a pipeline wait that runs out inside the kernel is reported through that buffer's status
    block and time limit, so ``buffer.check_status()`` raises and poisons it like any other failed device wait.

    Without ``out``, a product of few tiles and a long K is summed in up to 16 parts along K, in 32 bits and in an order that is fixed by M, N, K and
    ``num_sms``: the bits of a row can change with the batch that it is in.  The parts take a workspace of at most ``num_sms`` x 64 KB from
    PyTorch's allocator.  With ``out`` nothing is allocated and every sum is one chain along K: a row's bits depend on the row and the weights alone."""
    return _native.load().gemm_nt(a, b, None, None, None, out, num_sms, None, 0, None, _core_of(buffer))


def grouped_gemm_nt(a: torch.Tensor, b: torch.Tensor, tile_group: torch.Tensor, out: Optional[torch.Tensor] = None,
                    sfa: Optional[torch.Tensor] = None, sfb: Optional[torch.Tensor] = None, num_sms: int = 0, buffer=None,
                    tile_rows: Optional[torch.Tensor] = None, total_rows: int = 0) -> torch.Tensor:
    """Every 128-row tile ``t`` of ``a`` is multiplied by ``b[tile_group[t]]`` (``-1`` skips the tile).  bf16 operands,
    or e4m3 operands with ``sfa [M, K/128]`` and ``sfb [G, N/128, K/128]`` fp32 block scales.  ``buffer``: see
    :func:`gemm_nt`.  ``tile_rows`` int32 (of :func:`expert_tiles`): how many leading rows of every tile count; the kernel may leave
    the others unread and their results unwritten, which it does for e4m3 with ``N >= 256``.  ``total_rows``: how many token rows all
    tiles have together, at most or as expected, for a caller that knows it on the host; it chooses between kernels and changes no result.  With at
    most 56 per tile on average (and no more tiles than groups) the weights are streamed, which is up to a fifth faster; not known (0), the kernel
    for full tiles runs."""
    return _native.load().gemm_nt(a, b, sfa, sfb, tile_group, out, num_sms, None, 0, None, _core_of(buffer), tile_rows, total_rows)


def _plain(t: torch.Tensor) -> bool:
    """A tensor whose PyTorch statement nobody watches, so that a kernel of this library may take its place: no subclass, not wrapped
    by a function transform, no gradient or tangent to carry on, and nothing that records or intercepts operations is active.
    A native call would be invisible to those: ``torch.jit.trace`` and ``make_fx`` (a dispatch mode; fake tensors are another) would
    record the allocation of its results and not the launch that fills them."""
    return (type(t) in (torch.Tensor, torch.nn.Parameter) and not (t.requires_grad and torch.is_grad_enabled()) and
            torch.autograd.forward_ad._current_level < 0 and not torch.compiler.is_compiling() and not torch.jit.is_tracing() and
            torch._C._len_torch_dispatch_stack() == 0 and not torch._C._functorch.is_functorch_wrapped_tensor(t))


def _plain_cuda(t: torch.Tensor) -> bool:
    """:func:`_plain`, on the current GPU."""
    return t.is_cuda and t.device.index == torch.cuda.current_device() and _plain(t)


def quantize_weight_blocks(w: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """``w [G, N, K]`` -> (e4m3 ``[G, N, K]``, fp32 scales ``[G, ceil(N/128), ceil(K/128)]``), one scale per
    128 x 128 block (the weight format of DeepSeek-V3 style FP8 training).  One kernel for contiguous bf16 / fp32 weights on a
    GPU whose rows are whole 16-byte pieces; anything else takes the PyTorch statement below, which gives the same bits."""
    if (_plain_cuda(w) and w.dtype in (torch.bfloat16, torch.float32) and w.dim() == 3 and w.is_contiguous() and w.shape[2] % 8 == 0 and
            w.data_ptr() % 16 == 0):
        q, sf = _native.load().quantize_weight_blocks(w)
        return q, sf
    return quantize_weight_blocks_ref(w)


def quantize_weight_blocks_ref(w: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """The same cast stated with plain PyTorch operations (any device; what the kernel is tested against)."""
    G, N, K = w.shape
    nb, kb = (N + 127) // 128, (K + 127) // 128
    wp = torch.zeros(G, nb * 128, kb * 128, device=w.device, dtype=torch.float32)
    wp[:, :N, :K] = w
    blocks = wp.view(G, nb, 128, kb, 128)
    amax = blocks.abs().amax(dim=(2, 4)).clamp(1e-4)
    q = (blocks * (448.0 / amax)[:, :, None, :, None]).to(torch.float8_e4m3fn).view(G, nb * 128, kb * 128)[:, :N, :K].contiguous()
    return q, (amax / 448.0).contiguous()


def expert_segments(psum_expert_ends: torch.Tensor, num_rows: int, alignment: int = BLOCK_M) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """From the expand-layout segment ends of ``EPHandle.psum_num_recv_tokens_per_expert`` (segment ``i`` starts at
    ``align(end[i-1], alignment)``) -> (``tile_group int32 [ceil(num_rows / 128)]`` with -1 for tiles that hold no
    token, ``valid_row bool [num_rows]``, ``seg_off int32 [G + 1]`` aligned segment boundaries).  One kernel launch, no host
    synchronisation (CPU tensors take the plain PyTorch statement below)."""
    assert alignment % BLOCK_M == 0, 'expert segments must start on a tile boundary'
    if not psum_expert_ends.is_cuda:
        return expert_segments_ref(psum_expert_ends, num_rows, alignment)
    ends = psum_expert_ends if psum_expert_ends.dtype == torch.int32 else psum_expert_ends.to(torch.int32)
    return tuple(_native.load().expert_segments(ends.contiguous(), num_rows, alignment)[:3])


def expert_tiles(psum_expert_ends: torch.Tensor, num_rows: int, alignment: int = BLOCK_M):
    """:func:`expert_segments` with a fourth tensor, ``tile_rows int32 [ceil(num_rows / 128)]``: the token rows of every tile."""
    if not psum_expert_ends.is_cuda:
        tile_group, valid_row, seg_off = expert_segments_ref(psum_expert_ends, num_rows, alignment)
        padded = torch.zeros(tile_group.numel() * BLOCK_M, dtype=torch.bool)
        padded[:num_rows] = valid_row
        return tile_group, valid_row, seg_off, padded.view(-1, BLOCK_M).sum(1).to(torch.int32)
    assert alignment % BLOCK_M == 0, 'expert segments must start on a tile boundary'
    return tuple(_native.load().expert_segments(psum_expert_ends.to(torch.int32).contiguous(), num_rows, alignment))


def expert_tile_groups(psum_expert_ends: torch.Tensor, num_rows: int, alignment: int = BLOCK_M) -> Tuple[torch.Tensor, torch.Tensor]:
    """``(tile_group, valid_row)`` of ``expert_segments``."""
    return expert_segments(psum_expert_ends, num_rows, alignment)[:2]


def expert_segments_ref(psum_expert_ends: torch.Tensor, num_rows: int, alignment: int = BLOCK_M):
    """The same three tensors stated with plain PyTorch operations (what the kernel is tested against)."""
    ends = psum_expert_ends.to(torch.int64)
    aligned_ends = (ends + alignment - 1) // alignment * alignment
    starts = torch.cat([torch.zeros(1, dtype=torch.int64, device=ends.device), aligned_ends[:-1]])
    num_tiles = (num_rows + BLOCK_M - 1) // BLOCK_M
    tile_start = torch.arange(num_tiles, device=ends.device, dtype=torch.int64) * BLOCK_M
    grp = torch.searchsorted(aligned_ends, tile_start, right=True)
    grp_c = grp.clamp_max(ends.numel() - 1)
    has_rows = (grp < ends.numel()) & (tile_start < ends[grp_c]) & (tile_start >= starts[grp_c])
    tile_group = torch.where(has_rows, grp_c, torch.full_like(grp_c, -1)).to(torch.int32)
    rows = torch.arange(num_rows, device=ends.device, dtype=torch.int64)
    rgrp = torch.searchsorted(aligned_ends, rows, right=True).clamp_max(ends.numel() - 1)
    valid_row = (rows >= starts[rgrp]) & (rows < ends[rgrp])
    seg_off = torch.cat([torch.zeros(1, dtype=torch.int64, device=ends.device), aligned_ends]).to(torch.int32)
    return tile_group.contiguous(), valid_row, seg_off.contiguous()


def local_expand_plan(recv_idx: torch.Tensor, psum_aligned: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """For the output of a NON-expand dispatch made with ``expert_alignment=128``: ``recv_idx [rows, K]`` (local expert ids,
    -1 elsewhere) and ``EPHandle.psum_num_recv_tokens_per_expert`` (inclusive sums of the aligned counts) ->
    (``pos int32 [rows, K]``: the row of pair (row, k) in the per-expert (expand) layout, -1 if none; ``seg_end int32 [El]``:
    end of the token rows of every expert segment, the input of ``expert_segments``).  Rows of a segment are in received
    order, the same on every run."""
    if not recv_idx.is_cuda:
        return local_expand_plan_ref(recv_idx, psum_aligned)
    pos, seg_end = _native.load().local_expand_plan(recv_idx, psum_aligned.contiguous())
    return pos, seg_end


def local_expand_plan_ref(recv_idx: torch.Tensor, psum_aligned: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """The same two tensors stated with plain PyTorch operations (any device; what the kernels are tested against)."""
    El = psum_aligned.numel()
    ends = psum_aligned.to(torch.int64)
    idx = recv_idx.to(torch.int64)
    valid = (idx >= 0) & (idx < El)
    flat_e = torch.where(valid, idx, torch.full_like(idx, El)).reshape(-1)
    # stable sort by expert keeps the received (row-major) order inside every expert
    order = torch.sort(flat_e, stable=True).indices
    counts = torch.bincount(flat_e, minlength=El + 1)[:El]
    aligned = torch.cat([ends[:1], ends[1:] - ends[:-1]])
    starts = ends - aligned
    first = torch.cumsum(counts, 0) - counts                      # position of every expert's first pair in `order`
    sorted_e = flat_e[order]
    keep = sorted_e < El
    rank_in_e = torch.arange(order.numel(), device=idx.device) - first[sorted_e.clamp(max=El - 1)]
    pos = torch.full((idx.numel(),), -1, dtype=torch.int64, device=idx.device)
    pos[order[keep]] = (starts[sorted_e[keep]] + rank_in_e[keep])
    return pos.reshape(idx.shape).to(torch.int32), (starts + counts).to(torch.int32)


def local_expand_layout(recv_idx: torch.Tensor, psum_aligned: torch.Tensor, num_rows: int):
    """:func:`local_expand_plan` and :func:`expert_tiles` of its segments -> ``(pos, seg_end, tile_group, valid_row, seg_off,
    tile_rows)``; one launch when there are at most 1024 (row, k) pairs."""
    if not recv_idx.is_cuda:
        pos, seg_end = local_expand_plan_ref(recv_idx, psum_aligned)
        return (pos, seg_end, *expert_tiles(seg_end, num_rows))
    return tuple(_native.load().local_expand_layout(recv_idx, psum_aligned.contiguous(), num_rows))


def local_expand_copy(pos: torch.Tensor, x: torch.Tensor, num_out: int, sf: Optional[torch.Tensor] = None,
                      w: Optional[torch.Tensor] = None, valid_row: Optional[torch.Tensor] = None):
    """Writes every received row of ``x`` (and its scales ``sf [rows, G]`` / weights ``w [rows, K]``) to its expert rows ->
    ``[x_out [num_out, width], sf_out, w_out [num_out]]`` (only those asked for).  Alignment rows of the rows and scales are not written; their weights
    are zero (``valid_row`` of :func:`local_expand_layout`, if given, saves the launch that fills them)."""
    return _native.load().local_expand_copy(pos, x, num_out, sf, w, valid_row)


def local_reduce(pos: torch.Tensor, y: torch.Tensor, w: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``out[row] = sum_k w[pos[row, k]] * y[pos[row, k]]`` (``w``: one weight per expert row; plain sum without it) in fp32,
    rounded once to bf16."""
    return _native.load().local_reduce(pos, y, w, out)


def local_gather(pos: torch.Tensor, values: torch.Tensor) -> torch.Tensor:
    """``values[pos]`` for one fp32 value per expert row: fp32 ``[rows, K]``, zero where ``pos`` is -1."""
    return _native.load().local_gather(pos, values)


def per_token_cast_to_fp8(x: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """bf16 ``[rows, H]`` -> (e4m3 ``[rows, H]``, fp32 scales ``[rows, ceil(H / 128)]``), one kernel."""
    q, sf = _native.load().per_token_cast_to_fp8(x.contiguous())
    return q, sf


def swiglu_quant(h: torch.Tensor, keep_bf16: bool = False, valid_row: Optional[torch.Tensor] = None):
    """``h [rows, 2I]`` bf16 (gate | up) -> ``(e4m3 [rows, I], scales [rows, I/128][, bf16 activation])``.  Rows marked false in
    ``valid_row`` are skipped: nothing of them is read, and their results are not written."""
    return _native.load().swiglu_quant(h, keep_bf16, valid_row)


def gemm_kgrouped(a_t: torch.Tensor, b_t: torch.Tensor, k_off: torch.Tensor, num_sms: int = 0) -> torch.Tensor:
    """Weight gradients of a grouped layer in one launch: ``out[e] = a_t[:, k0:k1] @ b_t[:, k0:k1]^T`` with
    ``(k0, k1) = (k_off[e], k_off[e + 1])``; ``a_t [M, rows]``, ``b_t [N, rows]`` bf16 (the transposed activations and
    gradients, so that the reduction dimension = rows of the expert segment is contiguous), ``k_off`` int32
    ``[G + 1]`` multiples of 64 on the device.  -> bf16 ``[G, M, N]``; an expert without rows gets zeros.  For callers that hold
    transposed operands (:func:`moe_bwd_prep`, :func:`swiglu_bwd`, :func:`weighted_transpose` and :func:`dequant_transpose` write them);
    ``FusedMoE`` uses :func:`gemm_kgrouped_tn` on row-major ones."""
    return _native.load().gemm_kgrouped(a_t, b_t, k_off, num_sms)


def grouped_gemm_nn(a: torch.Tensor, b: torch.Tensor, tile_group: torch.Tensor, out: Optional[torch.Tensor] = None, num_sms: int = 0,
                    buffer=None) -> torch.Tensor:
    """Data gradient of a grouped layer on the forward weights as they are stored: every 128-row tile ``t`` of ``a [M, K]`` is
    multiplied by ``b[tile_group[t]]`` with ``b [G, K, N]`` (``-1`` skips the tile) -> bf16 ``[M, N]``.  The tensor core reads the
    N-contiguous operand through a transposing descriptor, so no transposed copy of the weights exists.  ``buffer``: see
    :func:`gemm_nt`."""
    return _native.load().grouped_gemm_nn(a, b, tile_group, out, num_sms, _core_of(buffer))


def gemm_kgrouped_tn(a: torch.Tensor, b: torch.Tensor, k_off: torch.Tensor, num_sms: int = 0) -> torch.Tensor:
    """:func:`gemm_kgrouped` on row-major operands: ``out[e] = a[k0:k1]^T @ b[k0:k1]`` with ``a [rows, M]``, ``b [rows, N]`` bf16.
    Every row of a segment enters the sum, so alignment rows must hold zeros in both (zero times a stale NaN is a NaN)."""
    return _native.load().gemm_kgrouped_tn(a, b, k_off, num_sms)


def swiglu_bwd_rows(d_act: torch.Tensor, h: torch.Tensor, valid_row: torch.Tensor, row_weight: torch.Tensor):
    """:func:`swiglu_bwd` with ``row_weight`` and row-major results -> ``(d_h [rows, 2I], activation [rows, I],
    d loss / d row_weight [rows])``; padding rows give zeros."""
    return _native.load().swiglu_bwd_rows(d_act, h, valid_row, row_weight)


def swiglu_bwd_rows_fp8(d_act: torch.Tensor, h: torch.Tensor, valid_row: torch.Tensor, row_weight: torch.Tensor):
    """:func:`swiglu_bwd_rows` with two more results, :func:`per_token_cast_to_fp8` of its ``d_h``: ``(d_h, activation,
    d loss / d row_weight, e4m3 d_h [rows, 2I], scales [rows, 2I / 128])``; ``I % 128 == 0``."""
    return _native.load().swiglu_bwd_rows(d_act, h, valid_row, row_weight, True)


def weighted_rows(g_rows: torch.Tensor, w: torch.Tensor, valid_row: torch.Tensor) -> torch.Tensor:
    """``g * w[:, None]`` as bf16 ``[rows, H]``; padding rows give zeros whatever they hold."""
    return _native.load().weighted_rows(g_rows, w, valid_row)


def dequant_rows(q: torch.Tensor, sf: torch.Tensor, valid_row: torch.Tensor, row_weight: Optional[torch.Tensor] = None) -> torch.Tensor:
    """e4m3 rows with 1 x 128 scales -> bf16 ``q * (scale * row_weight) [rows, H]``; padding rows give zeros."""
    return _native.load().dequant_rows(q, sf, valid_row, row_weight)


def segment_offsets(psum_expert_ends: torch.Tensor, alignment: int = BLOCK_M) -> torch.Tensor:
    """Expand-layout segment boundaries as ``int32 [G + 1]``: segment ``e`` covers rows ``[off[e], off[e + 1])``
    including its alignment padding.  Stays on the device."""
    return expert_segments(psum_expert_ends, 0, alignment)[2]


def moe_bwd_prep(g_rows: torch.Tensor, y: torch.Tensor, w: torch.Tensor, valid_row: torch.Tensor):
    """Backward of the weighted combine at the expert rows -> ``(g * w [rows, H], (g * w)^T [H, rows], sum(g * y) [rows])``;
    padding rows give zeros."""
    return _native.load().moe_bwd_prep(g_rows, y, w, valid_row)


def swiglu_bwd(d_act: torch.Tensor, h: torch.Tensor, valid_row: torch.Tensor, row_weight: Optional[torch.Tensor] = None):
    """Backward of ``silu(gate) * up`` -> ``(d_h [rows, 2I], d_h^T [2I, rows], activation^T [I, rows])``.  With
    ``row_weight [rows]`` the incoming gradient is taken as the gradient of the UNWEIGHTED activation: it is multiplied by
    the weight before it flows on, and ``sum_i d_act[r, i] * activation[r, i]`` (= d loss / d weight) is returned as a
    fourth tensor."""
    return _native.load().swiglu_bwd(d_act, h, valid_row, row_weight)


def weighted_transpose(g_rows: torch.Tensor, w: torch.Tensor, valid_row: torch.Tensor) -> torch.Tensor:
    """``(g * w[:, None])^T`` as bf16 ``[H, rows]`` with zero columns for padding rows."""
    return _native.load().weighted_transpose(g_rows, w, valid_row)


def dequant_transpose(q: torch.Tensor, sf: torch.Tensor, valid_row: torch.Tensor) -> torch.Tensor:
    """e4m3 rows with 1 x 128 scales -> bf16 ``(q * scale)^T [H, rows]``; padding rows give zeros."""
    return _native.load().dequant_transpose(q, sf, valid_row)
