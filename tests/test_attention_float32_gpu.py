"""The float32-arithmetic attention (csrc/attention_simt.cu): what a row's mask hides does not reach it."""
import pytest
import torch

from mini_llama_cpp_release_b200 import kernels
from test_kernels_gpu import DEV, DT, make_paged

pytestmark = pytest.mark.gpu


def _rows(kv, q, start, window=0):
    out = torch.empty_like(q)
    n, width = q.shape
    cu = torch.tensor([0, n], dtype=torch.int32, device=DEV)
    kernels.attention_simt(q, out, cu, torch.tensor([start], dtype=torch.int32, device=DEV), 1, n, width // kv.head_dim, kv,
                           kv.head_dim ** -0.5, window)
    return out


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,KV,hd", [(2, 2, 64), (4, 2, 80), (3, 3, 24), (1, 1, 320)])
def test_values_that_are_no_numbers_reach_no_row_that_does_not_see_their_tile(H, KV, hd, dtype):
    """A tile is 32 keys; the tokens begin at position 2, so that one warp's rows lie on both sides of a tile's edge."""
    g = torch.Generator().manual_seed(hd)
    start, n = 2, 66
    k, v = (torch.randn(n, KV, hd, generator=g) for _ in range(2))
    q = torch.randn(n - start, H * hd, generator=g).to(DT[dtype]).to(DEV)
    for window, spoiled, clean in ((0, slice(32, None), slice(0, 32 - start)),            # later tokens
                                   (8, slice(0, 32), slice(39 - start, None))):           # tokens the window has left behind
        want = _rows(make_paged([k], [v], DT[dtype]), q, start, window)
        assert torch.isfinite(want).all()
        for bad in (float("inf"), float("nan")):
            w = v.clone()
            w[spoiled] = bad
            got = _rows(make_paged([k], [w], DT[dtype]), q, start, window)
            assert torch.equal(got[clean], want[clean]) and not torch.isfinite(got).all()
