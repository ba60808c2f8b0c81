"""The package's own bfloat16 matrix product on tcgen05 tensor cores (``csrc/gemm_tcgen05.cu``).

``gemm_bf16(x, w)`` computes ``x w^T`` for ``x`` [M, K] and ``w`` [N, K].  Large M uses 128 x 256 tiles
with the activations on the 128-row side; M <= 64 swaps the operands so that the weight matrix
streams through the 128-row side once, with K split over several blocks when the weight matrix
alone has too few tiles to fill the GPU.  Epilogues: bfloat16 or float output with an optional bias,
and SwiGLU over a block-interleaved gate/up matrix (see ``interleave_gate_up``).
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Optional

import torch

from .basic import status_word
from .native import KernelError, check, i32, library, ptr, require_cuda, sm_count, stream_ptr

EPI_BF16, EPI_F32, EPI_SWIGLU, EPI_RELU_SQUARED = 0, 1, 2, 4
SWIGLU_BLOCK = 128  # the fused epilogue wants 128 gate rows followed by their 128 up rows, repeated
PAIR_MIN_ROWS = 128  # more rows than this: the pair kernel's 256-row tiles (when this package's kernels take a prompt-sized product at all)


def supported(x: torch.Tensor, w: torch.Tensor) -> bool:
    """Operands this kernel takes: bfloat16, K-contiguous, 16-byte aligned rows (strides multiples of 8 elements)."""
    return (x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.dim() == 2 and w.dim() == 2 and x.stride(1) == 1
            and w.stride(1) == 1 and x.stride(0) % 8 == 0 and w.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0
            and x.shape[1] == w.shape[1])


def interleave_gate_up(gate: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    """[I, H] gate and up matrices -> [2I, H] in blocks of 128 gate rows followed by the matching 128 up rows.
    I must be a multiple of 128."""
    inter, hidden = gate.shape
    if inter % SWIGLU_BLOCK:
        raise KernelError(f"the fused SwiGLU layout needs an intermediate size that is a multiple of {SWIGLU_BLOCK}, got {inter}")
    blocks = inter // SWIGLU_BLOCK
    return torch.stack([gate.view(blocks, SWIGLU_BLOCK, hidden), up.view(blocks, SWIGLU_BLOCK, hidden)], dim=1).reshape(2 * inter, hidden).contiguous()


def batch_tile_for(m: int) -> int:
    return 0 if m > 64 else (16 if m <= 16 else (32 if m <= 32 else 64))


def choose_splits(n: int, k: int, m: int = 64, sms: Optional[int] = None) -> int:
    """Split K so that the blocks fill the device (``sms`` multiprocessors, asked from the current device when absent):
    about two blocks per SM for up to 16 rows of activations (two blocks share an SM, one's start and epilogue pass under
    the other's stream, and the partial sums are small), about one per SM for more rows (the partial sums, ``splits`` times
    the output in float, cost more than the overlap gives); every split keeps at least 4 k-blocks."""
    sms = sms or sm_count()
    tiles = -(-n // 128)
    k_blocks = -(-k // 64)
    target = 2 * sms if m <= 16 else sms
    return max(1, min(target // tiles if tiles < target else 1, k_blocks // 4, 16))


FEW_ROWS = 16  # rows up to which csrc/few_rows.cu takes a product
FEW_BF16, FEW_F32, FEW_SWIGLU, FEW_PIECES = 0, 1, 2, 3


def takes_few_rows(x: torch.Tensor, w: torch.Tensor, gated_block: Optional[int] = None) -> bool:
    """Whether ``csrc/few_rows.cu`` takes a product of a few rows (with SwiGLU; without it :func:`pays_few_rows` also asks what else could): whole tiles of 16 rows of the matrix and of 64 of k, and a
    matrix small enough that the step is its waits, not its bytes.  Measured in chains of such products, one to eight rows: [896, 896] 4.1 -> 2.2 us, [2,048, 2,048] 3.7 -> 2.8, [4,096, 2,048] 5.9 -> 4.8, [9,728, 896] with SwiGLU
    8.1 -> 5.0, [16,384, 2,048] with SwiGLU 15.7 -> 14.3; beyond 20 MB only where k is short (a tile's sum over long k keeps few blocks busy: [4,096, 4,096] 6.9 -> 8.0),
    and not from some 70 MB on ([32,000, 2,048] 21.5 -> 24.6).  Nine to sixteen rows ask for twice the rows per unit: [2,048, 2,048] 3.9 -> 3.4, [4,096, 2,048] 6.1 -> 6.4,
    [9,728, 896] 8.9 -> 7.0.  ``gated_block``: with SwiGLU in the epilogue, over runs of that many gate rows."""
    m, (n, k) = x.shape[0], w.shape
    if m > FEW_ROWS or k % 64 or n % 16 or n * k > 68 << 19 or not supported(x, w) or not w.is_contiguous():
        return False
    if gated_block is not None and (n % 32 or gated_block < 8 or (n // 2) % gated_block or (gated_block != n // 2 and gated_block & (gated_block - 1))):
        return False
    megabytes = n * k / 2**19
    if m <= 8:
        return megabytes <= 20 or (k <= 2048 and megabytes <= 68)
    return megabytes <= 13 or (k < 2048 and megabytes <= 20)


def pays_few_rows(m: int, n: int, k: int, pieces: bool, sms: int) -> bool:
    """Whether a product without SwiGLU that ``csrc/few_rows.cu`` takes is also faster there than where else it would go: the split product of this file from k = 2,048 on, else
    the library.  ``pieces``: the caller adds up parts of k.  Measured at n = 16 to 32,768 by k = 64 to 16,384, 1 to 16 rows, this kernel over the other:

    * a block sums whole k for its tiles of 16 columns, so long k is a chain that splits do not have (8 rows, n 256: k 4,096 0.9, 8,192 1.28, 16,384 1.66), and tiles beyond two blocks to an SM are
      a second turn (8 rows, k 2,048: n 4,096 0.82, 5,120 1.06, 8,192 0.93), which only short k bears (n 10,240: k 256 0.9, 1,024 1.06);
    * where the split product's own blocks leave a second turn nearly empty it loses at any k (8 rows: [2,560, 2,048] 0.47, [1,536, 4,096] 0.69);
    * left in pieces, up to four parts of k fill the device from few tiles (8 rows: [896, 4,864] 0.78, [256, 16,384] 0.73; with more tiles than SMs they are whole sums: [2,560, 3,072] 1.26);
    * nine to sixteen rows ask for twice the rows per unit (16 rows: [1,024, 1,024] 0.70, [896, 4,864] 1.48 whole and 0.83 in pieces, [5,120, 1,024] 1.30)."""
    if n * k > (20 << 19 if k > 2048 else 68 << 19):  # bound by its bytes (takes_few_rows has the line); most products of a large model end here
        return False
    tiles, slots = n // 16, 2 * sms
    second_turn = k >= 2048 and sms < -(-n // 128) * choose_splits(n, k, m, sms) <= 1.5 * sms  # of the split product
    if pieces and k >= 2048:
        if second_turn:
            return True
        if m <= 8:
            return tiles <= sms and (k <= 6144 or 3 * tiles <= 2 * sms)
        return 8 * tiles < sms or (2 * tiles < sms and k <= 6144) or (tiles <= sms and k <= 2560)
    if m <= 8:
        if second_turn:
            return True
        if tiles <= slots:
            return k <= 3072 or (k <= 4096 and (2 * tiles < sms or 1.56 * tiles >= slots))
        if tiles <= 2 * slots:
            return k <= 1024 or (k <= 2560 and tiles >= 1.6 * slots)
        return k <= 256 and tiles <= 4 * slots
    if second_turn:
        return k <= 4096
    if 2 * tiles < sms:
        return k <= 2560
    return 128 <= k <= 1536 if tiles <= sms else 768 <= k <= 1536 and tiles <= slots


def few_rows(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, epilogue: int = FEW_BF16, block: int = 0, settled: bool = False):
    """``x w^T`` (+ bias) for up to 16 rows (``csrc/few_rows.cu``); :data:`FEW_SWIGLU` over gate and up rows in turn in runs of ``block``; :data:`FEW_PIECES`: a
    :class:`SplitSum`, its bias still to be added, or the whole sum where one block per tile is enough.
    ``settled``: the caller's word that no kernel still in flight writes ``w``; the product then fetches it while the kernel before still runs."""
    require_cuda(x, w, bias)
    m, k = x.shape
    n = w.shape[0]
    sms = sm_count(x.device)
    parts = 1
    if epilogue == FEW_PIECES:  # as many parts of k as there is room for two blocks to an SM, four units to a warp at the least
        parts = max(1, min(2 * sms // (n // 16), k // (64 * 8 * 2), 4))
        if parts == 1:
            epilogue = FEW_BF16
    if epilogue == FEW_PIECES:
        out = torch.empty((parts, m, n), dtype=torch.float32, device=x.device)
    else:
        out = torch.empty((m, n // 2 if epilogue == FEW_SWIGLU else n), dtype=torch.float32 if epilogue == FEW_F32 else torch.bfloat16, device=x.device)
    given = None if epilogue == FEW_PIECES else bias
    bias_f = given if given is not None and given.dtype == torch.float32 else None
    bias_h = given if given is not None and given.dtype == torch.bfloat16 else None
    check(library("few_rows").hb_few_rows(ptr(x), i32(x.stride(0)), ptr(w), ptr(bias_h), ptr(bias_f), ptr(out), i32(out.stride(-2)), i32(m), i32(n), i32(k), i32(epilogue),
                                          i32(block), i32(parts), i32(2 * sms), i32(1 if settled else 0), stream_ptr()), "few_rows")
    return SplitSum(out, bias, torch.bfloat16) if epilogue == FEW_PIECES else out


@dataclass
class SplitSum:
    """A product whose split-K partial sums have not been added up yet: ``partials`` [splits, M, N] float32, to be
    summed in split order, plus ``bias``, rounded to ``dtype``.  A consumer that can read the pieces itself (the fused
    residual add + norm) saves the kernel that would add them; everyone else calls :meth:`tensor`."""

    partials: torch.Tensor
    bias: Optional[torch.Tensor]
    dtype: torch.dtype

    @property
    def shape(self) -> tuple[int, int]:
        return tuple(self.partials.shape[1:])

    def tensor(self) -> torch.Tensor:
        splits, m, n = self.partials.shape
        out = torch.empty((m, n), dtype=self.dtype, device=self.partials.device)
        bias_f = self.bias if self.bias is not None and self.bias.dtype == torch.float32 else None
        bias_h = self.bias if self.bias is not None and self.bias.dtype == torch.bfloat16 else None
        check(library("gemm_tcgen05").hb_splitk_reduce(ptr(self.partials), i32(splits), i32(m), i32(n), ptr(out), i32(out.stride(0)),
                                                       i32(self.dtype == torch.float32), ptr(bias_f), ptr(bias_h), stream_ptr()), "splitk_reduce")
        return out


def gemm_bf16(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, epilogue: int = EPI_BF16,
              out: Optional[torch.Tensor] = None, splits: Optional[int] = None, leave_partials: bool = False):
    """``leave_partials``: when K is split, return a :class:`SplitSum` instead of adding the pieces up."""
    require_cuda(x, w, bias)
    if not supported(x, w):
        raise KernelError("gemm_bf16: operands must be bfloat16, K-contiguous, with 16-byte aligned rows")
    m, k = x.shape
    n = w.shape[0]
    out_cols = n // 2 if epilogue == EPI_SWIGLU else n
    out_dtype = torch.float32 if epilogue == EPI_F32 else torch.bfloat16
    if out is None:
        out = torch.empty((m, out_cols), dtype=out_dtype, device=x.device)
    if out.dtype != out_dtype or out.shape != (m, out_cols) or out.stride(1) != 1:
        raise KernelError("gemm_bf16: bad output tensor")
    bias_f = bias if bias is not None and bias.dtype == torch.float32 else None
    bias_h = bias if bias is not None and bias.dtype == torch.bfloat16 else None
    if bias is not None and bias_f is None and bias_h is None:
        raise KernelError("gemm_bf16: the bias is float32 or bfloat16")
    tile = batch_tile_for(m)
    if epilogue == EPI_SWIGLU:
        tile = 0  # the fused epilogue exists for the tile shape with activations on the 128-row side
    workspace = None
    if tile == 0:
        splits = 1
    else:
        splits = choose_splits(n, k, m) if splits is None else splits
        if splits > 1:
            workspace = torch.empty(splits * m * n, dtype=torch.float32, device=x.device)
    leave = int(leave_partials and workspace is not None and epilogue in (EPI_BF16, EPI_F32))
    lib = library("gemm_tcgen05")
    check(lib.hb_gemm_bf16(ptr(x), i32(x.stride(0)), ptr(w), i32(w.stride(0)), ptr(out), i32(out.stride(0)), ptr(bias_f), ptr(bias_h),
                           i32(m), i32(n), i32(k), i32(epilogue), i32(tile), i32(splits), ptr(workspace), i32(leave), ptr(status_word(x.device)),
                           stream_ptr()), "gemm_bf16")
    if leave:
        return SplitSum(workspace.view(splits, m, n), bias, out_dtype)
    return out


def gemm_pair_bf16(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, epilogue: int = EPI_BF16,
                   out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``x w^T`` on pairs of SMs (``csrc/gemm_pair_tcgen05.cu``: 256 x BN tiles, ``tcgen05.mma.cta_group::2``), for prompt-sized
    ``x``; the same operands and epilogues as :func:`gemm_bf16` in its tile shape."""
    require_cuda(x, w, bias)
    if not supported(x, w):
        raise KernelError("gemm_pair_bf16: operands must be bfloat16, K-contiguous, with 16-byte aligned rows")
    m, k = x.shape
    n = w.shape[0]
    out_cols = n // 2 if epilogue == EPI_SWIGLU else n
    out_dtype = torch.float32 if epilogue == EPI_F32 else torch.bfloat16
    if out is None:
        out = torch.empty((m, out_cols), dtype=out_dtype, device=x.device)
    if out.dtype != out_dtype or out.shape != (m, out_cols) or out.stride(1) != 1:
        raise KernelError("gemm_pair_bf16: bad output tensor")
    bias_f = bias if bias is not None and bias.dtype == torch.float32 else None
    bias_h = bias if bias is not None and bias.dtype == torch.bfloat16 else None
    if bias is not None and bias_f is None and bias_h is None:
        raise KernelError("gemm_pair_bf16: the bias is float32 or bfloat16")
    check(library("gemm_pair_tcgen05").hb_gemm_pair_bf16(ptr(x), i32(x.stride(0)), ptr(w), i32(w.stride(0)), ptr(out), i32(out.stride(0)), ptr(bias_f),
                                                         ptr(bias_h), i32(m), i32(n), i32(k), i32(epilogue), ptr(status_word(x.device)), stream_ptr()),
          "gemm_pair_bf16")
    return out
