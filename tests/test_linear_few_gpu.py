"""The float32 product (csrc/linear_simt.cu) at the edges of its tiles, chunks and stages: every output is the same sum in
the same order whichever kernel takes the step, so one shape's bits are another's."""
import pytest
import torch

from mini_llama_cpp_release_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,k", [(1, 4), (31, 252), (33, 256), (64, 260), (129, 320), (896, 4864), (5000, 516), (40, 5000), (4737, 64),
                                 (7, 255), (65, 18944), (33, 70000)])
def test_same_sum_whatever_the_rows(n, k):
    g = torch.Generator().manual_seed(n * 10007 + k)
    x = torch.randn(300, k, generator=g).to(DEV)
    w = torch.randn(n, k, generator=g).to(DEV)

    def product(rows, w=w):
        y = torch.full((rows, n), float("nan"), device=DEV)
        kernels.linear_simt(x[:rows], w, y)
        return y

    want = x.double() @ w.double().T
    whole = product(300)
    # a chunk's 256 terms and then the chunks: each addition rounds to 2^-24 of a partial sum, at most sqrt(K) times a few
    assert (whole - want).abs().max() <= 2.0 ** -24 * (min(k, 256) + k / 256) * 4.0 * k ** 0.5
    for rows in (1, 4, 5, 8, 9, 16, 17, 64, 65, 128):
        assert torch.equal(product(rows), whole[:rows]), rows
    # rows that no 16-byte load may touch take the general kernel
    odd = torch.empty(n * k + 1, device=DEV)[1:].view(n, k)
    odd.copy_(w)
    assert torch.equal(product(3, odd), whole[:3])


# (columns, K) of 17 to 64 rows on 148 SMs: tiles of 4 x 4 per thread up to 444 tiles of one or two chunks, single chunks below
# 78 % of a wave of 888 tiles, whole tiles from there on, single chunks again in the second wave
@pytest.mark.parametrize("n,k", [(1, 512), (500, 300), (28416, 512), (28417, 512), (44288, 512), (44353, 512), (56833, 300), (64, 600),
                                 (3000, 200), (30000, 256)])
def test_same_sum_in_every_form_of_17_to_64_rows(n, k):
    g = torch.Generator().manual_seed(n * 31 + k)
    x, w = torch.randn(65, k, generator=g).to(DEV), torch.randn(n, k, generator=g).to(DEV)

    def product(rows):
        y = torch.full((len(rows), n), float("nan"), device=DEV)
        kernels.linear_simt(rows, w, y)
        return y
    want = torch.cat([product(x[i:i + 13]) for i in range(0, 65, 13)])           # five steps of few rows
    for rows in (17, 33, 64, 65):
        assert torch.equal(product(x[:rows]), want[:rows]), rows
