"""Choice of the bfloat16 matrix-product kernel for a given shape.

* up to 64 rows (decode steps): the few-rows kernel (``gemm_skinny``: weights streamed once through registers) for up to 16
  rows of weights under 24 MB and K up to 4 096, else the weight-streaming tcgen05 kernel (``gemm_wstream``).  Both share a norm
  with the product on its other side and have the SiLU gate in their epilogue.  A decode step of the 8B layer sizes (eight layers) with the
  large products on ``gemm_wstream`` takes 839 / 903 / 896 / 1 006 us for 1 / 6 / 12 / 32 rows, with them on the library 963 / 999 / 990 /
  1 046; of the 0.6B sizes 1 077 us for 20 rows at 700 keys and 1 386 for 64 at 300 (1 326 and 1 451).  One product, weights cold, library / streamed
  / few rows: 8 x 4 096 x 4 096 11.9 / 7.8 / 8.6 us, 8 x 151 936 x 4 096 204 / 182 / 200, 8 x 24 576 x 4 096 34.4 / 35.5 / 37.4, 8 x 4 096 x 1 024
  4.8 / 4.3 / 2.5, 16 x 24 576 x 4 096 34.7 / 35.9 / 47.7; 64 x 6 144 x 4 096 11.3 / 13.5, so from 33 rows on products that share neither a norm
  nor a gate go to the library, and from 17 rows on those of them that it multiplies faster (``plain_takes_wstream``);
* 128 rows and more (prompt portions): the tcgen05 / TMA / TMEM kernel (``gemm_tcgen05``), with the SiLU gate in its
  epilogue for the gate/up projection — where the product has at least ``TCGEN05_MIN_TILES`` output tiles of
  128 x 128.  With fewer, every CTA walks the whole of K alone and the library, which splits K over more CTAs, measured
  1.3 to 2.7 times faster (2048 x 1024 x 2048: 8.8 us against 14.9), so those go to cuBLAS.  A product on the kernel that is followed by
  a norm adds to the residual itself; the line is the same: prompt steps of the 0.6B sizes with 2 400 / 2 919 / 3 500 / 4 096 tokens, whose
  output and down projections have 152 to 256 tiles, 4.11 / 4.81 / 5.72 / 6.07 ms on cuBLAS with norm kernels and 4.85 / 5.45 / 6.27 / 6.17 that
  way, with 4 700 / 8 192 (296 / 512 tiles) 8.02 / 14.83 and 7.96 / 14.41; of the 8B sizes 600 / 1 024 / 2 048 / 4 096 tokens (160 / 256 / 512 /
  1 024 tiles) 2.19 / 3.13 / 5.84 / 11.93 and 2.37 / 3.17 / 5.78 / 11.75;
* in between, and for K that is not a multiple of 8: the library product (cuBLAS via ``torch.mm``; the reference
  calls cuBLAS for every projection, csrc/ops/projection.cu:32-44), or the FMA kernel for shapes cuBLAS's
  tensor-core paths do not take.

``CUINFER_B200_GEMM=cublas`` sends every product of more than 16 rows to the library, ``CUINFER_B200_GEMM=tcgen05`` every
prompt-sized one that the kernel takes to the kernel (for comparisons); ``own`` (decode products of up to 16 rows on this
package's kernels) asks for what is always so.
"""
from __future__ import annotations

import torch

import os

from .. import kernels

# The library products of this package accumulate in 32 bits throughout: cuBLAS may otherwise reduce the partial sums
# of a split-K product in bfloat16 (torch allows that by default).
torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False

TCGEN05_MIN_ROWS = 128
TCGEN05_MIN_TILES = 296          # output tiles of 128 x 128 from which the tcgen05 kernel is chosen over the library
FEW_ROWS = 16
MANY_ROWS = 64                   # rows up to which the weight-streaming kernel is taken, and of products on their own
MANY_ROWS_PLAIN = 32
FUSED_NORM_MAX_K = 2048          # the norm prologue keeps 32-bit rows of all of K in shared memory: beyond this one CTA per SM
FEW_ROWS_LONG_K = 4096           # the few-rows kernel up to here, and for weights below
FEW_ROWS_MAX_BYTES = 24 << 20
_FORCE_CUBLAS = os.environ.get("CUINFER_B200_GEMM", "") == "cublas"
_FORCE_TCGEN05 = os.environ.get("CUINFER_B200_GEMM", "") == "tcgen05"


def few_rows_kernel(M: int, N: int, K: int) -> str:
    """Which kernel multiplies ``M <= 64`` rows with an [N, K] weight: "skinny", "wstream" or "library"."""
    if M <= FEW_ROWS and N * K * 2 < FEW_ROWS_MAX_BYTES and K <= FEW_ROWS_LONG_K:
        return "skinny"
    if M > MANY_ROWS_PLAIN and N * K * 2 >= FEW_ROWS_MAX_BYTES:
        return "library"          # (8B sizes, eight layers, 64 rows: a step 1 330 us on the library, 1 387 streamed; 48 rows the same on both)
    if kernels.gemm_wstream_supports(M, N, K) and not (M > FEW_ROWS and _FORCE_CUBLAS):
        return "wstream"
    return "skinny" if M <= FEW_ROWS else "library"


def plain_takes_wstream(M: int, N: int, K: int, out_dtype: torch.dtype) -> bool:
    """Whether rows that share neither a norm nor a gate stay on the weight-streaming kernel where ``few_rows_kernel`` says so.  Up
    to 16 rows always; to 32 rows where the library has to split K and add the parts up in a kernel of its own (at least two
    of K to a feature, or a few features), and for 32-bit rows; else the library is the faster one.  Inside decode steps of
    24 rows, streamed less library, us a product: 1 024 x 3 072 -2.4, 2 048 x 6 144 -1.6, 4 096 x 12 288 -2.8, 64 x 2 048 in 32
    bits -4.7, 32 768 x 4 096 in 32 bits -3; 4 096 x 1 024 +1.7, 6 144 x 1 024 +2.0, 12 288 x 2 048 +2.4, 2 048 x 2 048 between
    -0.8 and +1.4."""
    return M <= FEW_ROWS or (M <= MANY_ROWS_PLAIN and (K >= 2 * N or N <= 256 or out_dtype == torch.float32))


def wstream_takes(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """Whether the rows of both operands lie as ``gemm_wstream`` fetches them: apart, and on 16-byte boundaries."""
    K = x.shape[1]
    return all(t.stride(1) == 1 and t.stride(0) >= K and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 for t in (x, weight))


def takes_tcgen05(x: torch.Tensor, weight: torch.Tensor, fused: bool = False) -> bool:
    """``fused``: the product carries an epilogue (the SiLU gate) that the library call would need another kernel for;
    it stays on the tcgen05 kernel whatever its size."""
    return x.stride(1) == 1 and x.stride(0) % 8 == 0 and shape_takes_tcgen05(x.shape[0], weight, fused)


def shape_takes_tcgen05(M: int, weight: torch.Tensor, fused: bool = False) -> bool:
    """``takes_tcgen05`` for ``M`` dense rows."""
    N, K = weight.shape
    if not (M >= TCGEN05_MIN_ROWS and not _FORCE_CUBLAS and weight.stride(1) == 1 and weight.stride(0) % 8 == 0
            and kernels.gemm_tcgen05_supports(M, N, K)):
        return False
    if fused or _FORCE_TCGEN05 or K % 8 or N % 8:
        return True
    return -(-M // 128) * -(-N // 128) >= TCGEN05_MIN_TILES


def bf16_gated_matmul_nt(x: torch.Tensor, weight: torch.Tensor, gate=True) -> torch.Tensor | None:
    """silu(x gate^T) * (x up^T) for a weight of gate rows then up rows, in one tcgen05 kernel, when the shape is one
    it takes (prompt-sized, half of N a multiple of 8); None otherwise.  ``gate="gelu_tanh"``: the tanh form of GELU in
    the place of SiLU."""
    N = weight.shape[0]
    if x.dtype != torch.bfloat16 or weight.dtype != torch.bfloat16 or N % 16 or not takes_tcgen05(x, weight, fused=True):
        return None
    out = torch.empty((x.shape[0], N // 2), dtype=torch.bfloat16, device=x.device)
    kernels.gemm_tcgen05(x, weight, out, silu_pair=gate)
    return out


def bf16_matmul_nt(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor) -> None:
    """out[M, N] = x[M, K] @ weight[N, K]^T; x and weight bfloat16, out bfloat16 or float32."""
    M, K = x.shape
    N = weight.shape[0]
    if M <= MANY_ROWS_PLAIN and weight.stride(1) == 1 and x.stride(1) == 1:
        choice = few_rows_kernel(M, N, K)
        if (choice == "wstream" and plain_takes_wstream(M, N, K, out.dtype) and wstream_takes(x, weight)
                and out.stride(1) == 1 and out.stride(0) >= N):
            kernels.gemm_wstream(x, weight, out)
            return
        if choice == "skinny" and weight.is_contiguous() and kernels.gemm_skinny_supports(M, N, K):
            kernels.gemm_skinny(weight, out, act=x)
            return
    # (rows that lie inside wider rows are fine for the library as long as each starts on a 16-byte boundary)
    library_ok = (K % 8 == 0 and N % 8 == 0 and x.stride(1) == 1 and x.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0
                  and weight.is_contiguous())
    if takes_tcgen05(x, weight, fused=not library_ok):       # a product the library call cannot take stays on the kernel
        kernels.gemm_tcgen05(x, weight, out)
        return
    if library_ok:
        if out.dtype == torch.bfloat16:
            torch.mm(x, weight.t(), out=out)
            return
        if out.dtype == torch.float32:
            torch.mm(x, weight.t(), out_dtype=torch.float32, out=out)
            return
    kernels.gemm_generic(x, weight, out, constant_w=True)
