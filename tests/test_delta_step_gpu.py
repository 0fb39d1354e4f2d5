"""The gated delta rule's step of single tokens (csrc/recurrent.cu: delta_step_kernel) against the rule in 64 bits, at the edges
of its rows per warp and columns per block."""
from types import SimpleNamespace

import pytest
import torch

from mini_llama_cpp_release_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dim", [1, 8, 32, 33, 64, 100, 128, 129, 256])
@pytest.mark.parametrize("H,G,vdim", [(1, 1, 1), (4, 2, 32), (3, 1, 33), (6, 6, 64), (2, 1, 100)])
def test_single_tokens(dim, H, G, vdim):
    g = torch.Generator().manual_seed(dim * 1000 + vdim)
    n, slots = 3, [4, 0, 2]
    state = torch.randn(6, H * dim * vdim + 5, generator=g).to(DEV)[:, :H * dim * vdim]
    A_log, dt_bias = torch.randn(2, H, generator=g).to(DEV)
    before = state.clone()
    S = before[slots].double().view(n, H, dim, vdim)
    for _ in range(2):                                    # two steps in a row: the second reads what the first wrote
        qkv = torch.randn(n, 3 + 2 * G * dim + H * vdim, generator=g).to(DEV)
        gates = torch.randn(n, 2 * H + 1, generator=g).to(DEV)
        step = SimpleNamespace(n_seqs=n, n_tokens=n, max_q_len=1, slots=torch.tensor(slots, dtype=torch.int32, device=DEV),
                               cu_seqlens=torch.arange(n + 1, dtype=torch.int32, device=DEV))
        out = torch.full((n, H * vdim), float("nan"), device=DEV)
        kernels.gated_delta_rule(qkv, 3, 3 + G * dim, 3 + 2 * G * dim, gates, 1, 1 + H, A_log, dt_bias, state, step, H, G, dim, vdim, out)
        z = qkv.double()
        q, k = (z[:, c:c + G * dim].view(n, G, dim).repeat_interleave(H // G, 1) for c in (3, 3 + G * dim))
        v = z[:, 3 + 2 * G * dim:].view(n, H, vdim)
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dim ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        beta = torch.sigmoid(gates[:, 1:1 + H].double())[..., None]
        keep = torch.exp(-torch.exp(A_log.double()) * torch.nn.functional.softplus(gates[:, 1 + H:].double() + dt_bias.double()))
        S = keep[..., None, None] * S
        S = S + k[..., None] * (beta * (v - (S * k[..., None]).sum(2)))[:, :, None]
        want = (S * q[..., None]).sum(2).reshape(n, -1)
        # float32 sums of up to 256 terms, each within 2^-24 of itself, some of which cancel
        assert (out - want).abs().max() <= 2e-5 * max(1.0, float(want.abs().max()))
        assert (state[slots].double().view(n, H, dim, vdim) - S).abs().max() <= 2e-5 * float(S.abs().max())
    assert torch.equal(state[[1, 3, 5]], before[[1, 3, 5]])
