"""A product that adds into the stream (parts/linear.py: Linear.add_into): which kernel takes which rows, and what comes out on both sides of
every line between them."""
import pytest
import torch

from mini_llama_cpp_release_b200 import kernels
from mini_llama_cpp_release_b200.parts import linear


class _Runtime:
    n_sms = 148


def route(monkeypatch, n_tok, n_out, k):
    """("few" or "tcgen05", blocks that share the K range), without launching anything."""
    seen = []
    monkeypatch.setattr(kernels, "gemm_few", lambda x, w, out, epilogue, plan, *a, **kw: seen.append(("few", plan[4])))
    monkeypatch.setattr(kernels, "gemm_tcgen05", lambda x, w, out, epilogue, n_splits=1, *a, **kw: seen.append(("tcgen05", n_splits)))
    layer = linear.Linear(torch.empty(n_out, k, dtype=torch.bfloat16), _Runtime())
    layer.add_into(torch.empty(n_tok, k, dtype=torch.bfloat16), torch.empty(n_tok, n_out))
    assert len(seen) == 1
    return seen[0]


@pytest.mark.parametrize("n_out,k", [(512, 512), (640, 640), (1024, 256), (1536, 768), (2048, 832), (1024, 448)])
def test_a_whole_inner_size_is_added_by_one_block(monkeypatch, n_out, k):
    """17 to 32 rows: one plain add per element, so that the same bits come out every time."""
    for n_tok in (16, 17, 24):
        assert route(monkeypatch, n_tok, n_out, k) == ("few", 1), n_tok


def test_larger_products_leave_the_few_row_form_at_17_rows(monkeypatch):
    for n_out, k in ((896, 896), (896, 4864), (1536, 1536)):
        assert route(monkeypatch, 16, n_out, k)[0] == "few"
        for n_tok in (17, 32, 33, 64):
            assert route(monkeypatch, n_tok, n_out, k)[0] == "tcgen05"


@pytest.mark.parametrize("n_out,k", [(128, 8192), (64, 2048), (256, 1024), (512, 1024)])
def test_products_with_few_weights_stay_in_the_few_row_form(monkeypatch, n_out, k):
    for n_tok in (17, 32):
        assert route(monkeypatch, n_tok, n_out, k)[0] == "few"


@pytest.mark.parametrize("n_out,k,splits", [(256, 8192, 22), (512, 4096, 16), (128, 8192, 22), (896, 4864, 11), (1536, 1536, 6), (1536, 8960, 12),
                                            (2048, 2048, 5), (3584, 3584, 5), (1000, 136, 1), (896, 896, 7), (151936, 896, 1), (2, 8, 1)])
def test_blocks_that_share_an_inner_size(monkeypatch, n_out, k, splits):
    """33 to 64 rows: half of the SMs or seven K steps a block, whichever are more blocks; never an empty one."""
    for n_tok in (33, 64):
        assert route(monkeypatch, n_tok, n_out, k) == ("tcgen05", splits)
    steps = (k + 63) // 64
    for n_sms in (148, 132, 16, 1):
        for n_tok in (1, 2, 16, 17, 64):
            n = linear.add_split_count(n_out, k, n_tok, n_sms)
            assert 1 <= n <= steps and (n - 1) * -(-steps // n) < steps


@pytest.mark.gpu
@pytest.mark.parametrize("n_out,k", [(512, 512), (896, 896), (896, 4864), (208, 1000), (130, 1024), (1536, 768)])
@pytest.mark.parametrize("n_tok", [1, 16, 17, 24, 32, 33, 63, 64, 65])
def test_added_products_on_both_sides_of_the_lines(n_tok, n_out, k):
    """Against float64: sums of K products of 16-bit numbers in float32, each partial sum rounded by 2^-24 (3e-6 of the largest output, as
    for the kernels by themselves); a row beyond the output stays as it was; products that one block adds repeat bit for bit."""
    g = torch.Generator().manual_seed(n_tok + n_out + k)
    x = (torch.randn(n_tok, k, generator=g) * 0.5).bfloat16().cuda()
    layer = linear.Linear((torch.randn(n_out, k, generator=g) * 0.3).bfloat16().cuda(), _Runtime())
    before = torch.randn(n_tok + 1, n_out, generator=g).cuda()
    want = before[:n_tok].double() + x.double() @ layer.weight.double().T
    plan = layer.few_plan(n_tok, kernels.bindings.EPI_ADD)
    outs = []
    for _ in range(4):
        stream = before.clone()
        layer.add_into(x, stream[:n_tok])
        outs.append(stream)
        assert float((stream[:n_tok].double() - want).abs().max()) <= 3e-6 * float(want.abs().max())
        assert torch.equal(stream[n_tok], before[n_tok])
    if plan is not None and plan[4] == 1:
        assert all(torch.equal(o, outs[0]) for o in outs[1:])
    kernels.check_gemm_status(torch.device("cuda"))


@pytest.mark.gpu
@pytest.mark.parametrize("n_tok,n_out,k,splits", [(17, 896, 4864, 11), (24, 896, 4864, 10), (32, 896, 896, 7), (32, 208, 1000, 6), (33, 896, 4864, 11),
                                                  (63, 200, 1000, 8), (17, 130, 128, 1), (24, 300, 200, 2), (32, 1536, 1536, 12)])
def test_the_tcgen05_form_with_shared_inner_sizes(n_tok, n_out, k, splits):
    """Tiles of 32 and 64 tokens: a last split shorter than the others, splits of fewer K steps than threads that issue them, rows of w that
    are no multiple of 128.  Tolerance as above."""
    g = torch.Generator().manual_seed(n_tok + n_out + k)
    x = (torch.randn(n_tok, k, generator=g) * 0.5).bfloat16().cuda()
    w = (torch.randn(n_out, k, generator=g) * 0.3).bfloat16().cuda()
    before = torch.randn(n_tok + 1, n_out, generator=g).cuda()
    stream = before.clone()
    kernels.gemm_tcgen05(x, w, stream[:n_tok], kernels.bindings.EPI_ADD, splits)
    kernels.check_gemm_status(torch.device("cuda"))
    want = before[:n_tok].double() + x.double() @ w.double().T
    assert float((stream[:n_tok].double() - want).abs().max()) <= 3e-6 * float(want.abs().max())
    assert torch.equal(stream[n_tok], before[n_tok])
