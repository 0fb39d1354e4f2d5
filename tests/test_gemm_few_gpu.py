"""The product of a few rows (csrc/gemm_few.cu) at the edges of its tiles, units and token counts, against the same formula
in 64 bits; and the rule that hands products to it."""
import pytest
import torch

import plain_impl
from mini_llama_cpp_release_b200 import kernels
from mini_llama_cpp_release_b200.kernels import bindings
from mini_llama_cpp_release_b200.parts.rotary import neox_inv_freq
from test_kernels_gpu import DEV, close, make_paged

STORE, SILU, QKV, ADD = bindings.EPI_STORE, bindings.EPI_SILU_MUL, bindings.EPI_QKV, bindings.EPI_ADD
# float32 sums of K products in another order differ by at most K 2^-24 of the sum of the magnitudes, and the root of the
# mean square by a few units of the last place: far below 1e-5 of the largest output at these sizes
F32 = 1e-5
# shapes the kernel is compiled for: (units per warp, tiles at a time) by tiles of 8 tokens
SHAPES = {1: {(1, 1), (1, 2), (1, 3), (2, 1), (2, 2), (3, 1), (4, 1)}, 2: {(1, 1), (1, 2), (2, 1), (2, 2), (3, 1), (4, 1)},
          4: {(1, 1), (1, 2), (2, 1), (2, 2)}}


def test_every_plan_covers_its_product_with_a_compiled_shape():
    for n_sms in (148, 132, 16):
        for epi in (STORE, SILU, QKV, ADD):
            for n_tok in (1, 8, 9, 16, 17, 32):
                for k in list(range(64, 4200, 64)) + [4864, 8960, 18944]:
                    for n_out in (2, 16, 130, 896, 1152, 4608, 37888, 151936):
                        plan = bindings.gemm_few_plan(n_tok, n_out, k, epi, n_sms)
                        if plan is None:
                            continue
                        warps, uw, rt, blocks, splits = plan
                        per = -(-(k // 64) // splits)
                        assert 1 <= warps <= 16 and warps * uw >= per and (splits - 1) * per < k // 64
                        assert splits == 1 or epi == ADD
                        assert (uw, rt) in SHAPES[1 if n_tok <= 8 else 2 if n_tok <= 16 else 4] and blocks >= 1
                        tokens = 8 if n_tok <= 8 else 16 if n_tok <= 16 else 32
                        assert warps * rt * (uw * 2048 + tokens * 80) + 16 * tokens * 4 + 12 * tokens <= 227 * 1024
    for n_tok, k in ((33, 896), (8, 100), (8, 0), (0, 896)):
        assert bindings.gemm_few_plan(n_tok, 896, k, ADD, 148) is None


def operands(T, N, K, norm):
    g = torch.Generator().manual_seed(T * 1000 + N + K)
    w = (torch.randn(N, K, generator=g) * 0.3).to(torch.bfloat16)
    if not norm:
        x = (torch.randn(T, K, generator=g) * 0.5).to(torch.bfloat16)
        return x, w, None, x.double() @ w.double().t()
    x, gain = torch.randn(T, K, generator=g) * 3, 1 + 0.1 * torch.randn(K, generator=g)
    rms = 1 / (x.double().square().mean(-1, keepdim=True) + 1e-6).sqrt()
    return x, w, gain, ((x * gain).to(torch.bfloat16).double() @ w.double().t()) * rms


def run(x, w, out, epi, plan, gain, **kw):
    kernels.gemm_few(x.to(DEV), w.to(DEV), out, epi, plan, gain.to(DEV) if gain is not None else None, 1e-6, **kw)


# (rows, rows of w, columns, plan or None for the rule's): a last tile that is not full, fewer units than warps x units, one
# unit, several rounds of tiles per block, tiles left over in a round
CASES = [(1, 130, 64, None), (8, 1000, 896, (14, 1, 3, 5, 1)), (5, 37, 320, (2, 3, 1, 1, 1)), (7, 400, 896, (7, 2, 2, 4, 1)),
         (9, 130, 448, None), (16, 1000, 896, (14, 1, 2, 7, 1)), (13, 70, 704, (6, 2, 1, 2, 1)), (16, 64, 3584, (14, 4, 1, 3, 1)),
         (17, 130, 128, (2, 1, 2, 3, 1)), (32, 200, 896, (7, 2, 2, 3, 1)), (25, 33, 64, (1, 1, 1, 2, 1)), (3, 48, 3584, (14, 4, 1, 2, 1))]


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K,plan", CASES)
@pytest.mark.parametrize("norm", [False, True])
def test_few_rows_stored(T, N, K, plan, norm):
    x, w, gain, want = operands(T, N, K, norm)
    for dtype, tol in ((torch.float32, F32), (torch.bfloat16, 8e-3)):
        out = torch.full((T + 1, N), float("nan"), dtype=dtype, device=DEV)
        run(x, w, out[:T], STORE, plan or bindings.gemm_few_plan(T, N, K, STORE, 148), gain)
        close(out[:T].float(), want, tol)
        assert torch.isnan(out[T]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K,plan", [(T, N, K, p) for T, N, K, p in CASES if N % 2 == 0])
@pytest.mark.parametrize("norm", [False, True])
def test_few_rows_with_silu_mul(T, N, K, plan, norm):
    x, w, gain, want = operands(T, N, K, norm)
    out = torch.full((T, N // 2), float("nan"), dtype=torch.bfloat16, device=DEV)
    run(x, w, out, SILU, plan or bindings.gemm_few_plan(T, N, K, SILU, 148), gain)
    close(out.float(), torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2], 8e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K,plan", [(8, 896, 4864, None), (1, 896, 896, None), (16, 130, 1024, (4, 2, 1, 9, 2)), (3, 200, 128, (1, 2, 1, 4, 1)),
                                        (32, 896, 896, (7, 1, 1, 56, 2)), (5, 1000, 704, (4, 1, 2, 3, 3)), (8, 77, 448, (7, 1, 1, 5, 1))])
def test_few_rows_adding_into_the_stream(T, N, K, plan):
    x, w, _, want = operands(T, N, K, False)
    before = torch.randn(T, N, generator=torch.Generator().manual_seed(3))
    stream = before.clone().to(DEV)
    run(x, w, stream, ADD, plan or bindings.gemm_few_plan(T, N, K, ADD, 148), None)
    close(stream, before.double() + want, F32)


@pytest.mark.gpu
@pytest.mark.parametrize("H,KV,hd,T,K", [(6, 3, 32, 9, 192), (14, 2, 64, 8, 896), (3, 1, 16, 5, 64), (2, 2, 80, 30, 128), (2, 1, 256, 3, 3584), (3, 1, 18, 16, 128)])
@pytest.mark.parametrize("norm", [False, True])
def test_few_rows_with_qkv_epilogue(H, KV, hd, T, K, norm):
    x, w, gain, want = operands(T, (H + 2 * KV) * hd, K, norm)
    bias = torch.randn((H + 2 * KV) * hd, generator=torch.Generator().manual_seed(4))
    half = hd // 2
    within = torch.stack([torch.arange(half), torch.arange(half) + half], dim=1).reshape(-1)
    order = (torch.arange(H + 2 * KV)[:, None] * hd + within[None, :]).reshape(-1)
    q_lens = [T - T // 3, T // 3]
    lens = [q_lens[0] + 66, q_lens[1]]
    positions = torch.cat([torch.arange(n - m, n) for n, m in zip(lens, q_lens)]).to(torch.int32)
    tok_seq = torch.cat([torch.full((m,), b) for b, m in enumerate(q_lens)]).to(torch.int32)
    kv = make_paged([torch.zeros(n, KV, hd) for n in lens], [torch.zeros(n, KV, hd) for n in lens], torch.bfloat16)
    table = kernels.rope_table(neox_inv_freq(hd, 1e6).to(DEV), 512)
    q_out = torch.full((T, H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    run(x, w[order].contiguous(), q_out, QKV, bindings.gemm_few_plan(T, w.shape[0], K, QKV, 148), gain, bias=bias[order].contiguous().to(DEV),
        positions=positions.to(DEV), tok_seq=tok_seq.to(DEV), rope=table, q_heads=H, kv_heads=KV, head_dim=hd, kv=kv)
    full = (want + bias).float()
    pages = kv.page_table.cpu()
    got = [torch.stack([pool[1, int(pages[tok_seq[n], positions[n] // 64]), :, positions[n] % 64].float().cpu() for n in range(T)])
           for pool in (kv.k_pool, kv.v_pool)]
    close(q_out.float().view(T, H, hd), plain_impl.rope_neox(full[:, :H * hd].reshape(T, H, hd), positions, 1e6), 8e-3)
    close(got[0], plain_impl.rope_neox(full[:, H * hd:(H + KV) * hd].reshape(T, KV, hd), positions, 1e6), 8e-3)
    close(got[1], full[:, (H + KV) * hd:].reshape(T, KV, hd), 8e-3)
    assert torch.isnan(kv.k_pool[0].float()).all()


@pytest.mark.gpu
def test_few_rows_refuses_what_it_does_not_take():
    x, w = torch.zeros(8, 128, dtype=torch.bfloat16, device=DEV), torch.zeros(32, 128, dtype=torch.bfloat16, device=DEV)
    out = torch.empty(8, 32, device=DEV)
    for bad in ((1, 1, 1, 1, 1), (17, 1, 1, 1, 1), (2, 1, 1, 1, 2), (2, 1, 7, 1, 1), (2, 1, 1, 0, 1)):      # columns left out, too many warps, a split store, no such shape, no blocks
        with pytest.raises(kernels.KernelError, match="size"):
            kernels.gemm_few(x, w, out, STORE, bad)
    with pytest.raises(kernels.KernelError):
        kernels.gemm_few(x.float(), w, out, STORE, (2, 1, 1, 2, 1))
    big = torch.zeros(33, 128, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(kernels.KernelError, match="size"):
        kernels.gemm_few(big, w, torch.empty(33, 32, device=DEV), STORE, (2, 1, 1, 2, 1))


def test_short_inner_sizes_go_to_the_few_row_product_only_where_its_few_warps_keep_up():
    for n_tok, n_out, k, few in ((8, 1024, 128, True), (9, 1024, 128, False), (8, 1024, 64, False), (1, 1024, 64, True), (17, 1024, 256, True),
                                 (32, 1024, 256, False), (16, 4096, 256, False), (4, 4096, 256, True), (32, 1024, 512, True), (8, 4096, 4096, False)):
        assert (bindings.gemm_few_plan(n_tok, n_out, k, ADD, 148) is not None) is few, (n_tok, n_out, k)


@pytest.mark.gpu
@pytest.mark.parametrize("K", [64, 192, 320, 448, 896])
@pytest.mark.parametrize("T", [1, 8, 9, 16, 17, 32])
def test_adding_products_of_short_inner_sizes(T, K):
    for N in (16, 1000, 4100):
        plan = bindings.gemm_few_plan(T, N, K, ADD, 148)
        x, w, gain, want = operands(T, N, K, False)
        out = torch.ones(T, N, device=DEV)
        if plan is not None:
            run(x, w, out, ADD, plan, gain)
            close(out, want + 1, F32)
        store = bindings.gemm_few_plan(T, N, K, STORE, 148)
        if store is not None:
            run(x, w, out, STORE, store, gain)
            close(out, want, F32)
