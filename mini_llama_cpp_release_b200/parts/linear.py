"""y = x · Wᵀ for a weight stored [out, in] (src/matmul_optimized.cpp:40-54), the one
contraction every part is made of.

Which kernel runs is decided by the operand types and sizes, never by the model:
  * any float32 operand (the whole 32-bit path, or a tensor the checkpoint stores in
    32-bit while the engine computes in bfloat16): the float32 multiply-add kernel of
    csrc/linear_simt.cu.  No tensor-core mode takes part.
  * bfloat16 × bfloat16 of up to 32 rows, with an inner size that is a multiple of 64 and where
    `kernels.gemm_few_plan` has a plan (by rows, sizes and epilogue): the few-row product of
    csrc/gemm_few.cu, which also forms the RMS norm of its input on the way where a part may leave it
    to it (`of_norm`).
  * other bfloat16 × bfloat16 products with an inner size that is a multiple of 8: the tcgen05/TMA
    kernel of csrc/gemm_tcgen05.cu, when an epilogue is fused (Q/K/V with bias, rotation and
    cache write; gate/up with SiLU·mul), and for plain products of up to 64 rows (decoding),
    where the K range is split over blocks and the partial sums are left to the consumer.
  * plain bfloat16 products of more rows (prompts): the tokens-as-M tcgen05 kernels, one SM
    per tile (csrc/gemm_tcgen05_rows.cu) or, when tiles of 256 x 256 fill the GPU twice
    over, a pair of SMs per tile (csrc/gemm_tcgen05_pair.cu); where the product is a
    branch's last it adds into the float32 residual stream in its epilogue, with the K range
    shared out over blocks when the tiles alone would leave SMs idle.
  * bfloat16 products whose sizes those kernels do not take (an inner size that is no
    multiple of 8; in a prompt, a row count of W that is no multiple of 16): the library's
    product with float32 accumulation, as the reference calls cuBLAS for all of its linears
    (src/cuda_matmul.cpp:216-233).
"""
from __future__ import annotations

from typing import Optional

import torch

from .. import kernels
from .base import Runtime

SMALL_BATCH = 64          # up to this many rows a plain product runs on the tcgen05 kernel with split K
MAX_SPLITS = 8            # partial sums the consumer has to add
ADD_MAX_SPLITS = 24       # splits of a product that adds into the stream atomically (nobody has to add them up)
ADD_MAX_SPLITS_SOME = 10  # the same for 2 to 16 rows
ADD_SPLIT_STEPS = 7       # 64-element K steps that no split of 17 to 64 rows has more of, where the SMs allow it


def split_count(n_out: int, k: int, n_tok: int, n_sms: int, max_splits: int = 0) -> int:
    """How many blocks share the K range of a skinny product: enough to occupy the SMs, each
    with at least two 64-element K steps."""
    if n_tok > SMALL_BATCH:
        return 1
    row_tiles = (n_out + 127) // 128
    k_blocks = (k + 63) // 64
    s = max(1, min(n_sms // max(1, row_tiles), k_blocks // 2, max_splits or MAX_SPLITS))
    per = (k_blocks + s - 1) // s
    return (k_blocks + per - 1) // per


def add_split_count(n_out: int, k: int, n_tok: int, n_sms: int) -> int:
    """The blocks that share the K range of a product of up to 64 rows that adds into the stream.  More blocks stream the weights
    faster, but every block adds its part with one atomic per row and column, and its blocks are SMs on which the kernel after it
    cannot start early to ask for its own weights.

    Up to 16 rows, measured on whole decode steps of 24 and 28 layers on a B200, caps of 8 / 10 / 12 / 24: 0.733 / 0.710 / 0.717 /
    0.722 ms at 8 rows and 1.271 against 1.300 ms (10 against 24) at 16 rows of the Qwen2-1.5B sizes, but 0.735 / 0.703 / 0.704 /
    0.683 ms at one row; at the 7B sizes the cap does not bind.

    17 to 64 rows: as many as fill half of the SMs, and more while a block has more than seven K steps.  Whole decode steps, us:
    896 x 4,864 at the 0.5B sizes with 10 / 11 / 13 / 19 splits 20 rows 655 / 636 / 644 / 641, 48 rows 719 / 704 / 702 / 714, 64 rows
    741 / 735 / 730 / 725; 1,536 x 1,536 at the 1.5B sizes with 4 / 6 / 8 / 12 20 rows 1,193 / 1,174 / 1,172 / 1,190, 64 rows 1,266 /
    1,270 / 1,269 / 1,292.  us in a chain, weights from memory, 32 rows (17 to 64 alike): 2,048 x 2,048 5 splits 3.56, 8 3.92; 4,096 x
    1,024 2 3.56, 4 4.01; 1,024 x 8,192 16 5.12, 9 5.63; 256 x 8,192 22 3.20, 12 4.18; 512 x 4,096 16 2.92, 11 3.18; 1,536 x 8,960
    (the SMs allow 12) 6.55, 6 7.27."""
    if n_tok <= 16:
        cap = ADD_MAX_SPLITS if n_tok < 2 else ADD_MAX_SPLITS_SOME
    else:
        tiles = (n_out + 127) // 128
        cap = min(ADD_MAX_SPLITS, max(n_sms // (2 * tiles), -(-((k + 63) // 64) // ADD_SPLIT_STEPS)))
    return split_count(n_out, k, n_tok, n_sms, max_splits=cap)


class Linear:
    def __init__(self, weight: torch.Tensor, runtime: Runtime):
        assert weight.dim() == 2
        self.weight = weight.contiguous()
        self.runtime = runtime
        self.out_features, self.in_features = weight.shape
        self.tensor_core_ok = (weight.dtype == torch.bfloat16 and self.in_features % 8 == 0
                               and self.weight.data_ptr() % 16 == 0)

    def nbytes(self) -> int:
        return self.weight.numel() * self.weight.element_size()

    def few_plan(self, n_rows: int, epilogue: int = 0):
        """The plan of the few-row product (csrc/gemm_few.cu), or None where another kernel takes these rows."""
        if n_rows > kernels.FEW_ROWS or not self.tensor_core_ok:
            return None
        return kernels.gemm_few_plan(n_rows, self.out_features, self.in_features, epilogue, self.runtime.n_sms)

    def of_norm(self, stream: torch.Tensor, gain: torch.Tensor, eps: float) -> torch.Tensor:
        """float32 [n, out]: the product of the float32 stream's RMS norm, for a row count that has a `few_plan`."""
        out = self.runtime.empty(stream.shape[0], self.out_features, dtype=torch.float32)
        kernels.gemm_few(stream, self.weight, out, kernels.bindings.EPI_STORE, self.few_plan(stream.shape[0]), gain, eps)
        return out

    def can_add_into_stream(self, n_rows: int) -> bool:
        """Whether `add_into` has a kernel for these operands: the few-row and tcgen05 products (plain or atomic adds for
        few rows, adding copies by TMA for more), else the library's product with the stream as the matrix it adds to."""
        return self.tensor_core_ok

    def add_into(self, x: torch.Tensor, stream: torch.Tensor) -> None:
        """stream (float32 [n, out]) += x · Wᵀ.  Few rows: the few-row product where it has a plan, else the weights-as-M tcgen05
        product, the K range shared out over as many blocks as is useful.  More rows: the tokens-as-M tcgen05 product, with a K split when its tiles alone
        would leave SMs idle (the library's product only for a row count that kernel does not take: no multiple of
        16).  Either way the stream is updated in the product's epilogue, so the norm that follows has one tensor to
        read, not two."""
        m = x.shape[0]
        if m > SMALL_BATCH and kernels.gemm_rows_takes(m, self.out_features, self.in_features):
            kernels.gemm_prompt(x, self.weight, stream, kernels.bindings.EPI_ADD, n_sms=self.runtime.n_sms)
            return
        if m > SMALL_BATCH:
            kernels.library_gemm(x, self.weight, stream, accumulate=True)
            return
        if (plan := self.few_plan(m, kernels.bindings.EPI_ADD)) is not None:
            kernels.gemm_few(x, self.weight, stream, kernels.bindings.EPI_ADD, plan)
            return
        splits = add_split_count(self.out_features, self.in_features, m, self.runtime.n_sms)
        kernels.gemm_tcgen05(x, self.weight, stream, kernels.bindings.EPI_ADD, splits, n_sms=self.runtime.n_sms)

    def __call__(self, x: torch.Tensor, out_dtype: torch.dtype = torch.float32, partial_ok: bool = False) -> torch.Tensor:
        """[n, out] in `out_dtype`; with `partial_ok` possibly float32 partial sums [slices, n, out]
        whose sum over the first axis is the product."""
        assert x.dim() == 2 and x.shape[1] == self.in_features, (x.shape, self.weight.shape)
        rt = self.runtime
        m = x.shape[0]
        if x.dtype == torch.float32 or self.weight.dtype == torch.float32:
            out = rt.empty(m, self.out_features, dtype=out_dtype)
            kernels.linear_simt(x, self.weight, out)
            return out
        kernels.require_cuda(x)
        if (plan := self.few_plan(m)) is not None:
            out = rt.empty(m, self.out_features, dtype=out_dtype)
            kernels.gemm_few(x, self.weight, out, kernels.bindings.EPI_STORE, plan)
            return out
        if self.tensor_core_ok and m <= SMALL_BATCH:
            splits = split_count(self.out_features, self.in_features, m, rt.n_sms) if (partial_ok and out_dtype == torch.float32) else 1
            out = rt.empty(splits, m, self.out_features, dtype=out_dtype)
            kernels.gemm_tcgen05(x, self.weight, out, kernels.bindings.EPI_STORE, splits, n_sms=rt.n_sms)
            return out if splits > 1 else out[0]
        out = rt.empty(m, self.out_features, dtype=out_dtype)
        if self.tensor_core_ok and kernels.gemm_rows_takes(m, self.out_features, self.in_features):
            kernels.gemm_prompt(x, self.weight, out, kernels.bindings.EPI_STORE, n_sms=rt.n_sms)
        else:
            kernels.library_gemm(x, self.weight, out)
        return out
