"""Which keys a row of the tcgen05 prompt attention sees, where a tile of 64 keys is cut: by the diagonal, by a window's edge, by first keys
that stay visible beside it, by a chunk's first key; whole prompts and steps that continue a cached part."""
import math

import pytest
import torch

from mini_llama_cpp_release_b200 import kernels
from test_kernels_gpu import DEV, make_paged

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window,keep,chunk", [(0, 0, 0), (1, 0, 0), (63, 0, 0), (64, 5, 0), (65, 64, 0), (100, 70, 0), (0, 0, 64), (0, 0, 97)])
@pytest.mark.parametrize("n,m", [(1, 1), (64, 64), (65, 65), (193, 130), (300, 37)])
@pytest.mark.parametrize("H,KV,hd", [(14, 2, 64), (4, 2, 128)])
def test_what_a_row_sees(H, KV, hd, n, m, window, keep, chunk):
    """Against float64; probabilities and outputs are rounded to 16 bits (2^-9 each), as in the kernel's other tests."""
    g = torch.Generator().manual_seed(n + m + hd)
    k, v = (torch.randn(n, KV, hd, generator=g).bfloat16().float() for _ in range(2))
    q = torch.randn(m, H, hd, generator=g).bfloat16().float()
    kv = make_paged([k], [v], torch.bfloat16, seed=n)
    out = torch.full((m, H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    cu = torch.tensor([0, m], dtype=torch.int32, device=DEV)
    start = torch.tensor([n - m], dtype=torch.int32, device=DEV)
    kernels.attention_tcgen05(q.bfloat16().view(m, H * hd).to(DEV), out, cu, start, 1, m, H, kv, 1.0 / math.sqrt(hd), window,
                              keep_first=keep, chunk=chunk)
    kernels.check_gemm_status(DEV)
    i, j = torch.arange(n - m, n)[:, None], torch.arange(n)[None]
    seen = j <= i
    if window:
        seen &= (i - j < window) | (j < keep)
    if chunk:
        seen &= i // chunk == j // chunk
    k, v = (t.double().repeat_interleave(H // KV, 1).transpose(0, 1) for t in (k, v))
    s = (q.double().transpose(0, 1) @ k.transpose(1, 2) / math.sqrt(hd)).masked_fill(~seen, -math.inf)
    want = (torch.softmax(s, -1) @ v).transpose(0, 1).reshape(m, H * hd)
    assert float((out.double().cpu() - want).abs().max()) <= 1e-2 * float(want.abs().max())
