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


# x of 60.2 MB: its pieces are shared by consecutive blocks; of half as many tokens W's are
LONG, LONG_K = 30100, 1000


@pytest.mark.parametrize("epilogue", [bindings.EPI_STORE, bindings.EPI_SILU_MUL, bindings.EPI_ADD])
@pytest.mark.parametrize("form,width", [("rows", 128), ("rows", 224), ("pair", 256)])
def test_both_walks_give_the_same_bits(form, width, epilogue):
    """An output's sum runs over K in the same order wherever its tile stands: all tokens at once and half of them at a time agree."""
    n_out, half = 208, LONG // 2
    g = torch.Generator().manual_seed(5)
    x = (torch.randn(LONG, LONG_K, generator=g) * 0.5).bfloat16().to(DEV)
    w = (torch.randn(n_out, LONG_K, generator=g) * 0.1).bfloat16().to(DEV)
    run = kernels.gemm_tcgen05_pair if form == "pair" else kernels.gemm_tcgen05_rows
    before = torch.randn(LONG, n_out // 2 if epilogue == bindings.EPI_SILU_MUL else n_out, device=DEV)
    whole, parts = before.clone(), before.clone()
    run(x, w, whole, epilogue, width, 1)
    for part in (slice(0, half), slice(half, LONG)):
        run(x[part], w, parts[part], epilogue, width, 1)
    kernels.check_gemm_status(torch.device(DEV))
    assert torch.equal(whole, parts)
    if epilogue == bindings.EPI_STORE:
        want = x.double() @ w.double().T
        assert float((whole.double() - want).abs().max()) <= TOL * float(want.abs().max())


def test_both_walks_of_the_qkv_product_give_the_same_bits():
    H, KV, hd, half = 4, 1, 64, LONG // 2
    g = torch.Generator().manual_seed(6)
    x = (torch.randn(LONG, LONG_K, generator=g) * 0.5).bfloat16().to(DEV)
    w = (torch.randn((H + 2 * KV) * hd, LONG_K, generator=g) * 0.1).bfloat16().to(DEV)
    pos = torch.arange(LONG, dtype=torch.int32, device=DEV)
    seq = torch.zeros(LONG, dtype=torch.int32, device=DEV)
    rope = torch.randn(LONG, hd // 2, 2, generator=g).to(DEV)
    pages = (LONG + 63) // 64
    table = torch.arange(pages, dtype=torch.int32, device=DEV).view(1, pages)
    got = []
    for cuts in ((0, LONG), (0, half, LONG)):
        kv = kernels.KVView(*(torch.zeros(1, pages, KV, 64, hd, dtype=torch.bfloat16, device=DEV) for _ in range(2)), 0, table, 64, KV, hd)
        q = torch.empty(LONG, H * hd, dtype=torch.bfloat16, device=DEV)
        for a, b in zip(cuts, cuts[1:]):
            kernels.gemm_tcgen05_rows(x[a:b], w, q[a:b], bindings.EPI_QKV, positions=pos[a:b], tok_seq=seq[a:b], rope=rope, q_heads=H,
                                      kv_heads=KV, head_dim=hd, kv=kv)
        got.append((q, kv.k_pool, kv.v_pool))
    kernels.check_gemm_status(torch.device(DEV))
    assert all(torch.equal(a, b) for a, b in zip(*got)) and bool(got[0][1].any()) and bool(got[0][2].any())
