"""Plain dense matrix products: few rows as a stream over the weight, large float32 products on the tensor cores with their
operands in parts, the others through the library (cuBLAS via torch.mm).

The reference's dense products (``Bundle::mm``, src/bundle.rs:644-683) are a
library call as well: ndarray's ``dot`` over matrixmultiply or cblas.  Weights
stay in the checkpoint's ``(out, in)`` layout; the product is ``rows @ W^T``
with float32 accumulation and a float32 result.  In float32 mode the library's
reduced precision matrix modes (TF32, bf16 reductions) are switched off and that
is checked at every call.
"""
from __future__ import annotations

from functools import partial
from typing import Optional

import torch

from ..csrc import ops

_ONE_TILE: dict[tuple[str, int], tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]] = {}
STREAM_ROWS = 8           # up to this many rows a dense product is a stream over the weight (experts_stream.cu; float32: rows_f32.cu); beyond,
                          # each item's rows of x are as many bytes as its weights and the library's product is faster (measured at
                          # 12 to 32 rows on a B200: 14 to 25 us against 11 for MiniMax-M2's projections)
# A float32 weight of up to this many entries is streamed by the dense products' kernel, a larger one by the experts' (both in rows_f32.cu).
# The number of rows has no say: the two add a row's products in different orders, and a sequence's results shall not depend on how many
# others are in its step.  The line lies where no number of rows is slower by the first than by the second; microseconds for 1, 4 and 8
# rows by the second | the first: 65536 x 1024 weights 42 54 77 | 41 44 60, 21845 x 3072 43 56 63 | 41 43 45; beyond, 65536 x 3072
# 113 141 163 | 120 125 126, 131072 x 2048 157 183 194 | 158 188 232, 200064 x 3072 338 417 469 | 362 383 419.
DENSE_ROWS_ENTRIES = 1 << 26
STREAM_FEATURES = 65536   # beyond this many output features the library product is at the memory roofline anyway


# A float32 product runs on the tensor cores, each operand as two float16 parts (products_f32.cu), from SPLIT_PRODUCTS multiply-adds,
# SPLIT_ROWS rows and SPLIT_TILES tiles of 128 x 128 results on.  Below, the pass over the weight for its scales (half of the bytes of
# a product of few rows), the launches or the idle SMs cost more than the products save.  Measured on a B200 with weights that are not in
# L2, microseconds, the library's float32 product | this one with its scales and parts: 200064 x 3072 weights, 9 rows 853 | 1218, 32 rows
# 896 | 772, 48 rows 1397 | 820; 32768 x 4096, 32 rows 265 | 229, 64 rows 341 | 209; 8192 x 3072, 48 rows (2^30.2) 97 | 71, 64 rows 97 | 72,
# 96 rows 128 | 76, 700 rows 613 | 160; 3072 x 6144, 64 rows 151 | 94, 128 rows (24 tiles) 169 | 103, 256 rows 250 | 112; 2048 x 2048, 128 rows
# (2^29) 52 | 47, 256 rows 58 | 49, 512 rows 88 | 53; 1024 x 1024, 1,024 rows (2^30) 48 | 39, 2,048 rows 86 | 40; 256 x 3072, 2,048 rows 82 | 67.
# (The lines lie where they were with the kernel before; by these figures they would lie at 2^30, 32 rows and 16 tiles.)
SPLIT_ROWS = 48
SPLIT_TILES = 32
SPLIT_PRODUCTS = 1 << 31
LONG_STEP = 16384         # tokens of the longest step that the generation loop runs


def split_products_reach(needs) -> bool:
    """Whether a step of up to LONG_STEP tokens may run a float32 product with one of these matrices (or with all of them as one weight)
    as split products: a part whose products stay below that does not ask for their kernels."""
    sizes = [need.shape[0] * need.shape[1] for need in needs if len(need.shape) == 2 and ops.products_f32_take(need.shape[1])]
    return sum(sizes) * LONG_STEP >= SPLIT_PRODUCTS


def one_tile(device: torch.device, rows: int):
    key = (str(device), rows)
    if key not in _ONE_TILE:
        zero = torch.zeros(1, dtype=torch.int32, device=device)
        _ONE_TILE[key] = (zero, zero.clone(), torch.ones(1, dtype=torch.int32, device=device),
                          torch.tensor([0, rows], dtype=torch.int32, device=device))
    return _ONE_TILE[key]


def require_true_float32() -> None:
    """Switch off every reduced-precision mode of the library's float32 matrix products.  (This library's own products split their
    operands where they run on tensor cores, and are held to 64-bit sums: products_f32.cu, tf32_parts.cuh.)"""
    torch.backends.cuda.matmul.allow_tf32 = False
    torch.backends.cudnn.allow_tf32 = False
    torch.set_float32_matmul_precision("highest")
    if hasattr(torch.backends.cuda.matmul, "allow_bf16_reduced_precision_reduction"):
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
    if hasattr(torch.backends.cuda.matmul, "allow_fp16_reduced_precision_reduction"):
        torch.backends.cuda.matmul.allow_fp16_reduced_precision_reduction = False


def full_sums() -> None:
    """Products with a bfloat16 result add in float32 to the end and round once."""
    if hasattr(torch.backends.cuda.matmul, "allow_bf16_reduced_precision_reduction"):
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False


def split_products_pay(rows: int, weight: torch.Tensor) -> bool:
    return (rows * weight.numel() >= SPLIT_PRODUCTS and rows >= SPLIT_ROWS
            and -(-rows // 128) * -(-weight.shape[0] // 128) >= SPLIT_TILES)


def float32_kernels_read(rows: torch.Tensor, weight: torch.Tensor, out: Optional[torch.Tensor]) -> bool:
    """Whether the float32 kernels may read these operands and write this result: matrices that fit together and lie in one piece
    from a 16-byte boundary on.  The library takes the others, or refuses them."""
    return (rows.dim() == 2 and weight.dim() == 2 and rows.shape[1] == weight.shape[1] and rows.numel() > 0
            and (out is None or (out.shape == (rows.shape[0], weight.shape[0]) and out.dtype == torch.float32 and out.is_contiguous()))
            and rows.is_contiguous() and weight.is_contiguous() and rows.data_ptr() % 16 == 0 and weight.data_ptr() % 16 == 0)


def linear(rows: torch.Tensor, weight: torch.Tensor, out: Optional[torch.Tensor] = None, rounded: bool = False,
           split: bool = True, weight_final: bool = False) -> torch.Tensor:
    """rows [T, in] @ weight[out, in]^T -> float32 [T, out]; ``split``: whether a large float32 product may run as split products
    on the tensor cores; with ``rounded`` (bfloat16 rows only) the float32 sums rounded once
    to bfloat16, for a reader that takes its operands in that type anyway.  ``weight_final``: the weight was complete before the
    kernel before this product in the stream began, so that a product of few rows may read it while that one still runs."""
    if rounded:
        if rows.dtype != torch.bfloat16 or weight.dtype != torch.bfloat16 or not rows.is_cuda or out is not None:
            raise RuntimeError(f"a rounded matrix product of {rows.dtype} rows with a {weight.dtype} weight on {rows.device}")
        with ops.timed(f"library_mm_bf16[{weight.shape[0]}x{weight.shape[1]}]"):
            return torch.mm(rows, weight.t())
    if not rows.is_cuda:
        raise RuntimeError("fieldrun_b200 runs on a CUDA device only; a CPU tensor reached a matrix product")
    if rows.dtype != weight.dtype:
        raise RuntimeError(f"matrix product of {rows.dtype} rows with a {weight.dtype} weight")
    if rows.dtype == torch.float32:
        if torch.backends.cuda.matmul.allow_tf32 or torch.get_float32_matmul_precision() != "highest":
            raise RuntimeError("a float32 matrix product was asked for while TF32 is allowed")
        few = rows.shape[0] <= STREAM_ROWS
        many = split and rows.shape[0] >= SPLIT_ROWS and split_products_pay(rows.shape[0], weight)
        if (few or many) and float32_kernels_read(rows, weight, out) \
                and (ops.rows_f32_takes(rows.shape[1]) if few else ops.products_f32_take(rows.shape[1])):
            result = out if out is not None else torch.empty((rows.shape[0], weight.shape[0]), dtype=torch.float32, device=rows.device)
            if few:
                if weight.numel() > DENSE_ROWS_ENTRIES:
                    tile_expert, tile_row0, num_tiles, offsets = one_tile(rows.device, rows.shape[0])
                    ops.rows_f32(weight.unsqueeze(0), rows, None, tile_expert, tile_row0, num_tiles, offsets, 1, result, paired=False)
                else:
                    ops.dense_rows_f32(weight, rows, result, weights_final=weight_final)
            else:
                parts = torch.empty((2, *rows.shape), dtype=torch.float16, device=rows.device)
                scale = torch.empty(rows.shape[0], dtype=torch.float32, device=rows.device)
                ops.products_f32(weight.unsqueeze(0), ops.weight_scales(weight), rows, parts, scale, result)
            return result
        with ops.timed(f"library_mm_f32[{weight.shape[0]}x{weight.shape[1]}]"):
            if out is None:
                return torch.mm(rows, weight.t())
            return torch.mm(rows, weight.t(), out=out)
    count, inner = rows.shape
    features = weight.shape[0]
    if count <= STREAM_ROWS and inner % 32 == 0 and features % 16 == 0 and features <= STREAM_FEATURES \
            and rows.is_contiguous() and weight.is_contiguous():
        # few rows: the weight is the traffic; stream it once through the kernel that streams expert weights,
        # the dense layer being a single expert whose rows are all the rows
        tile_rows = 8 if count <= 8 else 16 if count <= 16 else 32
        tile_expert, tile_row0, num_tiles, offsets = one_tile(rows.device, count)
        result = out if out is not None else torch.empty((count, features), dtype=torch.float32, device=rows.device)
        if ops.weight_stream_takes(features, inner, paired=False):
            # the lists of this one tile never change, so a weight that does not either may be on its way before the rows are ready
            ops.weight_stream(weight.view(1, features, inner), rows, None, tile_expert, tile_row0, num_tiles, offsets, 1,
                              tile_rows, result, paired=False, lists_final=weight_final)
        else:
            ops.expert_gemm_mma(weight.view(1, features, inner), rows, None, tile_expert, tile_row0, num_tiles, offsets, 1,
                                tile_rows, result, paired=False, **ops.stream_shape(1, features, inner, tile_rows))
        return result
    with ops.timed(f"library_mm[{features}x{inner}]"):
        result = torch.mm(rows, weight.t(), out_dtype=torch.float32)
    if out is None:
        return result
    out.copy_(result)
    return out


# The product with a part's own weight, which a step finds as it was loaded (see Part.load).
part_linear = partial(linear, weight_final=True)
