"""Prompts through memories that decay per head (csrc/gla_chunks.cu) against the same tokens one at a time (the step of
single tokens, csrc/linear_attention.cu), which the per-design tests check against plain loops."""
from types import SimpleNamespace

import pytest
import torch

from mini_llama_cpp_release_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SLOTS = [4, 0, 2]


def _step(lens):
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).int()
    return SimpleNamespace(n_seqs=len(lens), n_tokens=sum(lens), max_q_len=max(lens), cu_seqlens=cu.to(DEV),
                           slots=torch.tensor(SLOTS[:len(lens)], dtype=torch.int32, device=DEV))


def _both(lens, width, n_state, H_vdim, run):
    """Outputs and states of one step with all tokens, and of one step per position; the state starts as noise."""
    g = torch.Generator().manual_seed(sum(lens) * 31 + width)
    rows = [torch.randn(n, width, generator=g).to(DEV) for n in lens]
    start = (torch.rand(6, n_state + 3, generator=g) * 0.5).to(DEV)
    whole = start.clone()
    out = torch.empty(sum(lens), H_vdim, device=DEV)
    run(torch.cat(rows), whole[:, :n_state], _step(lens), out)
    single = start.clone()
    parts = [torch.empty(n, H_vdim, device=DEV) for n in lens]
    for t in range(max(lens)):
        # sequences that have ended take an earlier token once more, into a slot of their own
        live = [i for i, n in enumerate(lens) if n > t]
        step = _step([1] * len(live))
        step.slots = torch.tensor([SLOTS[i] for i in live], dtype=torch.int32, device=DEV)
        o = torch.empty(len(live), H_vdim, device=DEV)
        run(torch.cat([rows[i][t:t + 1] for i in live]), single[:, :n_state], step, o)
        for j, i in enumerate(live):
            parts[i][t] = o[j]
    assert torch.equal(whole[1], start[1]) and torch.equal(whole[5], start[5])        # slots of no sequence
    return out, torch.cat(parts), whole, single


def _close(a, b, tol):
    assert torch.isfinite(a).all()
    assert float((a.double() - b.double()).norm() / b.double().norm()) <= tol


# A sum of up to 64 + dim products in another order, each within 2^-24 of itself: 1e-5 leaves room for terms that cancel
TOL = 1e-5
SHAPES = [(2, 24, 40), (1, 200, 65), (3, 64, 100), (2, 130, 33), (6, 128, 256)]
LENS = [[33], [64], [65, 1, 34], [128, 63, 129], [191, 200, 2]]


@pytest.mark.parametrize("H,dim,vdim", SHAPES)
@pytest.mark.parametrize("lens", LENS)
def test_constant_decay(H, dim, vdim, lens):
    decay = torch.tensor([0.3, 0.995, 0.9, 1.0, 0.6, 0.05][:H], device=DEV)
    gain = torch.ones(H * vdim, device=DEV)

    def run(x, state, step, out):
        kernels.decay_attention(x, 0, 2 * H * dim + H * vdim, decay, gain, 1e-5, 1.0, state, step, H, dim, vdim, out)
    a, b, sa, sb = _both(lens, 2 * H * dim + 2 * H * vdim, H * dim * vdim, H * vdim, run)
    _close(a, b, TOL)
    _close(sa, sb, TOL)


@pytest.mark.parametrize("H,dim,vdim", SHAPES)
@pytest.mark.parametrize("lens", LENS)
def test_exponential_gates(H, dim, vdim, lens):
    bias, gain = torch.randn(2, H).to(DEV), torch.ones(H * vdim, device=DEV)
    cols, c = [], 0
    for size in (H * dim, H * dim, H * vdim, H * vdim, H, H):
        cols.append(c)
        c += size

    def run(x, state, step, out):
        kernels.matrix_memory(x, *cols, bias[0], bias[1], 12.0, gain, 1e-5, state, step, H, dim, vdim, out)
    a, b, sa, sb = _both(lens, c, H * dim * (vdim + 1) + H, H * vdim, run)
    _close(a, b, 1e-4)               # divided by |n·q|, a sum that cancels
    _close(sa, sb, TOL)


@pytest.mark.parametrize("lens", LENS)
def test_state_space_groups(lens):
    H, G, N, vdim = 6, 2, 72, 48
    inner, n_conv = H * vdim, H * vdim + 2 * G * N
    vec = torch.randn(3, H).to(DEV)
    gain = torch.ones(inner, device=DEV)

    def run(x, state, step, out):
        proj, xbc = x[:, :inner + H].contiguous(), x[:, inner + H:].contiguous()
        kernels.state_space(proj, 0, inner, xbc, inner, inner + G * N, vec[0], vec[1], vec[2], gain, 1e-5, 1, state, step, H, G, N, vdim, out)
    a, b, sa, sb = _both(lens, inner + H + n_conv, inner * N, inner, run)
    _close(a, b, TOL)
    _close(sa, sb, TOL)


def test_a_value_that_is_not_a_number_reaches_no_earlier_token():
    H, dim, vdim, n, bad = 2, 32, 40, 100, 70
    x = torch.randn(n, 2 * H * dim + 2 * H * vdim, generator=torch.Generator().manual_seed(1)).to(DEV)
    decay, gain = torch.tensor([0.9, 0.99], device=DEV), torch.ones(H * vdim, device=DEV)
    outs = []
    for spoil in (False, True):
        rows = x.clone()
        if spoil:
            rows[bad, 2 * H * dim:2 * H * dim + H * vdim] = float("inf")
        out = torch.empty(n, H * vdim, device=DEV)
        kernels.decay_attention(rows, 0, 2 * H * dim + H * vdim, decay, gain, 1e-5, 1.0, torch.zeros(6, H * dim * vdim, device=DEV),
                                _step([n]), H, dim, vdim, out)
        outs.append(out)
    assert torch.equal(outs[0][:bad], outs[1][:bad]) and not torch.isfinite(outs[1][bad:]).any()
