"""The experts' product of a few (token, choice) pairs (csrc/gemm_few_grouped.cu) against 64-bit products."""
import pytest
import torch

from mini_llama_cpp_release_b200 import kernels
from mini_llama_cpp_release_b200.kernels.bindings import EPI_SILU_MUL, EPI_STORE

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _plan(ids, E, tile):
    n, top = ids.shape
    rows = kernels.moe_plan_rows(n * top, E, tile)
    row_of, src = torch.empty(n, top, dtype=torch.int32, device=DEV), torch.empty(rows, dtype=torch.int32, device=DEV)
    tiles = torch.empty(rows // tile, dtype=torch.int32, device=DEV)
    kernels.moe_plan(ids, E, tile, row_of, src, tiles)
    return row_of, src, tiles


@pytest.mark.parametrize("n,top,E", [(1, 1, 1), (8, 1, 8), (4, 2, 5), (3, 3, 3), (16, 1, 2), (8, 2, 40), (1, 16, 16)])
@pytest.mark.parametrize("hidden,inter", [(64, 8), (128, 72), (1536, 448), (320, 5120), (2048, 4480)])
def test_experts_of_few_pairs(n, top, E, hidden, inter):
    assert kernels.gemm_few_grouped_takes(n * top, hidden, hidden)
    g = torch.Generator().manual_seed(n * 100 + E + hidden)
    ids = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(n)]).int().to(DEV)
    x = torch.randn(n, hidden, generator=g).to(DEV).bfloat16()
    w = (torch.randn(E, 2 * inter, hidden, generator=g) * hidden ** -0.5).to(DEV).bfloat16()
    tile = 8 if n * top <= 8 else 16
    row_of, src, tiles = _plan(ids, E, tile)
    n_sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = src.numel()
    # gathered, gated
    act = torch.full((rows, inter), float("nan"), device=DEV, dtype=torch.bfloat16)
    kernels.gemm_few_grouped(x, src, w, tiles, tile, act, EPI_SILU_MUL, n_sms)
    gu = torch.einsum("tjok,tk->tjo", w.double()[ids.long()], x.double())
    want = torch.nn.functional.silu(gu[..., 0::2]) * gu[..., 1::2]
    got = act[row_of.long()].double()
    # the result's rounding to 16 bits, and float32 sums whose products the gate multiplies
    assert (got - want).abs().max() <= 2.0 ** -8 * want.abs().max() and float((got - want).norm() / want.norm()) <= 2.0 ** -8
    # rows as they lie, plain, float32
    if kernels.gemm_few_grouped_takes(n * top, hidden, inter):
        down = (torch.randn(E, hidden, inter, generator=g) * inter ** -0.5).to(DEV).bfloat16()
        y = torch.full((rows, hidden), float("nan"), device=DEV)
        kernels.gemm_few_grouped(act, None, down, tiles, tile, y, EPI_STORE, n_sms)
        want = torch.einsum("tjok,tjk->tjo", down.double()[ids.long()], act[row_of.long()].double())
        assert float((y[row_of.long()].double() - want).norm() / want.norm()) <= 1e-6


def test_what_it_does_not_take():
    assert not kernels.gemm_few_grouped_takes(17, 128, 128) and not kernels.gemm_few_grouped_takes(8, 128, 96)
    assert not kernels.gemm_few_grouped_takes(8, 128, 5184) and not kernels.gemm_few_grouped_takes(0, 128, 128)
