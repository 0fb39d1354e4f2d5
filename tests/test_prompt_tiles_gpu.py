"""Prompt products whose float32 tiles leave by TMA and whose tiles are walked from either operand (csrc/gemm_rows_common.cuh): token and
column counts at the edges of a warp's 32 x 32 tile, of a block's tile and of a pair's, W's rows in fewer and in more than the tokens."""
import pytest
import torch

from mini_llama_cpp_release_b200 import kernels
from mini_llama_cpp_release_b200.kernels import bindings

pytestmark = pytest.mark.gpu
DEV = "cuda"
# float32 sums of K products of 16-bit numbers, in another order than float64's: K terms, each rounded by 2^-24 of a partial sum
TOL = 2e-5


def _operands(n_tok, n_out, k):
    g = torch.Generator().manual_seed(n_tok * 7 + n_out + k)
    x = (torch.randn(n_tok, k, generator=g) * 0.5).bfloat16().to(DEV)
    w = (torch.randn(n_out, k, generator=g) * 0.1).bfloat16().to(DEV)
    return x, w, x.double() @ w.double().T


@pytest.mark.parametrize("n_tok,n_out,k", [(65, 16, 72), (100, 144, 64), (257, 1040, 200), (300, 80, 1000), (1000, 912, 136), (129, 2000, 520)])
@pytest.mark.parametrize("form,width", [("rows", 128), ("rows", 160), ("rows", 224), ("rows", 256), ("pair", 128), ("pair", 160), ("pair", 224), ("pair", 256)])
def test_added_and_stored_tiles(form, width, n_tok, n_out, k):
    x, w, want = _operands(n_tok, n_out, k)
    run = kernels.gemm_tcgen05_pair if form == "pair" else kernels.gemm_tcgen05_rows
    before = torch.randn(n_tok + 1, n_out, device=DEV)                # a row beyond the output must stay as it is
    splits = 2 if k > 500 else 1
    out = before.clone()
    run(x, w, out[:n_tok], bindings.EPI_ADD, width, splits)
    got = (out[:n_tok].double() - before[:n_tok].double())
    # the added sum is rounded to float32 beside the old value
    assert float((got - want).abs().max()) <= TOL * float(want.abs().max()) + 2.0 ** -22 * float(before.abs().max() + want.abs().max())
    assert torch.equal(out[n_tok], before[n_tok])
    out = before.clone()
    run(x, w, out[:n_tok], bindings.EPI_STORE, width, 1)
    assert float((out[:n_tok].double() - want).abs().max()) <= TOL * float(want.abs().max())
    assert torch.equal(out[n_tok], before[n_tok])
    kernels.check_gemm_status(torch.device(DEV))
