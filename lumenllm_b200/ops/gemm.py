"""bfloat16 matrix products with float32 accumulation.

The tcgen05 / TMA kernels (csrc/gemm_tc.cu) do the work for every shape: two SMs a tile for
prompts, a weight-streaming orientation with k split for decode and short prompts. A product
may come back as S partial sums [S, M, N] for the consumer to add, or be added to the residual
stream in place. The library product (cuBLAS through torch, as the reference uses cuBLASLt:
crates/aegisllm-cuda/src/cuda/runtime/cublaslt.rs:57-165) stands only where a row of the
operands is not a multiple of 16 bytes, which the TMA cannot address. Weights reach the
tensor-core kernels in tiled form (kernels.tile_weight), made once when the model is built.
"""
from __future__ import annotations

import torch

from . import kernels as K
from .native import KernelError

torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
torch.backends.cuda.matmul.allow_tf32 = False
torch.backends.cudnn.allow_tf32 = False


def takes_tc(x: torch.Tensor, w) -> bool:
    """A weight in tiled form goes to the tensor-core kernels (it exists only where its rows are
    multiples of 16 bytes); a plain tensor is a weight they cannot address."""
    return isinstance(w, K.TiledWeight) and x.shape[1] % 8 == 0 and x.data_ptr() % 16 == 0


def gemm_bf16(x: torch.Tensor, w: torch.Tensor, split_ok: bool = False, add_to=None,
              col_scale=None):
    """x bfloat16 [M, K], w bfloat16 [N, K] (tiled, or a plain tensor) -> float32 [M, N]; with split_ok possibly
    [S, M, N] partial sums that the consumer adds. With add_to (float32 [M, N]) the product
    may instead be added to it in place, its columns times col_scale where given, where the kernel
    for this shape can do that; None is returned then, and the caller has nothing left to add (or to
    multiply: a product that is returned has not been)."""
    if x.dtype != torch.bfloat16 or w.dtype != torch.bfloat16:
        raise KernelError(f"gemm_bf16: expected bfloat16 operands, got {x.dtype} and {w.dtype}")
    if not x.is_cuda:
        raise KernelError("gemm_bf16: no CPU path exists")
    if not x.is_contiguous():
        x = x.contiguous()
    if takes_tc(x, w):
        if (add_to is not None and add_to.is_contiguous() and add_to.data_ptr() % 16 == 0
                and K.gemm_tc_adds(x.shape[0], w.shape[0])):
            return K.gemm_tc(x, w, add_to=add_to, col_scale=col_scale)
        part = K.gemm_tc(x, w)
    else:
        if isinstance(w, K.TiledWeight):
            raise KernelError(f"gemm_bf16: activations [{x.shape[0]}, {x.shape[1]}] do not fit a tiled weight "
                              f"{w.shape} (rows of 16 bytes, 16-byte aligned)")
        return torch.mm(x, w.t(), out_dtype=torch.float32)
    if part.shape[0] == 1:
        return part[0]
    return part if split_ok else part.sum(dim=0)


def gate_up_in_one(rows: int, width: int, k: int) -> bool:
    """Whether a gate/up product [rows, k] x [width, k]^T goes through its activation in the product's epilogue. Up to 128 rows
    the product streams the weights with k split, which the epilogue cannot have (at 100 rows of the 8B shape 41 + 6 us against
    56 us), and up to 255 its one row of tiles is part empty (160 rows: 57 us and the activation behind it against 73); 256 rows
    fill it, and more than 512 have tiles enough. Between, two things count. Below 56
    tiles of 256 x 256 the float32 product can split k over idle SMs, which pays for long k and few tiles; from
    56 on the two-SM kernel's epilogue, with its divisions, is longer than that of the float32 sums, which shows where k is
    short or the last wave of tiles is not full. us, one kernel / two, width x k:
    300 rows 1,024 x 1,024 7.7 / 9.3; 6,144 x 1,024 10.4 / 18.5; 4,096 x 2,048 14.0 / 15.5; 2,816 x 2,048 12.9 / 16.9;
    1,024 x 4,096 21.1 / 13.9; 4,096 x 4,096 23.4 / 19.4; 4,096 x 8,192 42.6 / 28.5; 6,144 x 8,192 45.2 / 41.8;
    8,192 x 1,024 18.4 / 15.8; 16,384 x 1,024 29.1 / 24.0; 10,240 x 2,048 33.4 / 31.3; 16,384 x 2,048 35.0 / 35.1;
    24,576 x 4,096 78.2 / 82.8; 448 rows 12,288 x 4,096 53.8 / 56.3, 8,192 x 4,096 33.9 / 32.3."""
    if rows <= 256 or rows > 512:
        return rows >= 256
    tiles = (rows + 255) // 256 * ((width + 255) // 256)
    if tiles >= 56:
        return k >= 2048 and (tiles >= 128 or (tiles >= 80 and rows > 352))
    return k <= 2048 or (tiles >= 36 and k <= 6144) or K.gemm_tc_splits(rows, width, k) == 1


def gemm_gate_up_silu(x: torch.Tensor, w_interleaved, act="silu"):
    """silu(gate) * up (or, `act` "gelu", gelu_tanh(gate) * up) in bfloat16 [M, I] from x [M, K] and a weight [2I, K] whose rows
    alternate gate_i, up_i, in ONE kernel where that is the faster way (gate_up_in_one); else None, and the
    caller takes the float32 product with the activation kernel behind it."""
    if takes_tc(x, w_interleaved) and gate_up_in_one(x.shape[0], w_interleaved.shape[0], x.shape[1]):
        return K.gemm_tc(x if x.is_contiguous() else x.contiguous(), w_interleaved,
                         silu_interleaved=True, act=act)
    return None


def gemm_gelu(x: torch.Tensor, w):
    """gelu_tanh(x w^T) in bfloat16 [M, N] in ONE kernel where the two-SM product takes the shape (its epilogue has
    the float32 sums at hand; 2,048 x 8,192 x 2,048: 58 us, 81 with the activation kernel behind); else None, and the
    caller takes the float32 product with the activation kernel behind it."""
    if takes_tc(x, w) and K.gemm_tc_gelu_takes(x.shape[0], w.shape[0]):
        return K.gemm_tc(x if x.is_contiguous() else x.contiguous(), w, gelu=True)
    return None
