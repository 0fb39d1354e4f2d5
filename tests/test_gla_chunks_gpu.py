"""Prompts through memories that decay per head (csrc/gla_chunks.cu) against the same tokens one at a time (the step of
single tokens, csrc/linear_attention.cu), which the per-design tests check against plain loops; both against the recurrences in
64 bits; and the rule that chooses between the chunks and the walk."""
import math
from types import SimpleNamespace

import pytest
import torch

from mini_llama_cpp_release_b200 import kernels
from mini_llama_cpp_release_b200.kernels import bindings

DEV = "cuda:0"
SLOTS = [4, 0, 2]


def test_the_rule_takes_the_form_that_was_measured_to_be_the_sooner():
    """(tokens of the long runs, how many, single tokens beside them) of 6 heads of 128 x 256 and of 2 of 24 x 40."""
    def pays(H, dim, vdim, length, runs, ones):
        rows = 4                                                    # mlc_gla_rows on 148 SMs
        while 8 * rows < dim:
            rows *= 2
        base = (runs + ones) * H * math.ceil(vdim / 32)
        while rows > 2 and base * math.ceil(dim / (8 * rows)) < 296:
            rows //= 2
        return bindings.gla_chunks_pay(runs + ones, length * runs + ones, length, H, dim, vdim, rows)
    for steps, want in (([(33, 1, 0), (64, 1, 0), (128, 1, 0), (48, 1, 31), (64, 1, 127), (256, 1, 127), (33, 4, 60)], False),
                        ([(512, 1, 0), (2048, 1, 0), (64, 16, 0), (64, 64, 0), (256, 1, 7), (2048, 1, 127), (1500, 3, 0)], True)):
        assert all(pays(6, 128, 256, *s) is want for s in steps)
    assert not pays(2, 24, 40, 128, 64, 0) and pays(2, 24, 40, 1024, 1, 0)


@pytest.fixture
def chunks(monkeypatch):
    """The chunks, however short the runs are; returns a check that a step of these lengths takes them."""
    monkeypatch.setattr(bindings, "gla_chunks_pay", lambda *a: True)

    def taken(lens, H=2, dim=32, vdim=40):
        plan = bindings._head_decay_plan(_step(lens), sum(lens), H, dim, vdim, torch.device(DEV))
        return (plan[2] is not None) == (max(lens) > 32)
    return taken


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


@pytest.mark.gpu
@pytest.mark.parametrize("H,dim,vdim", SHAPES)
@pytest.mark.parametrize("lens", LENS)
def test_constant_decay(H, dim, vdim, lens, chunks):
    decay = torch.tensor([0.3, 0.995, 0.9, 1.0, 0.6, 0.05][:H], device=DEV)
    gain = torch.ones(H * vdim, device=DEV)

    def run(x, state, step, out):
        kernels.decay_attention(x, 0, 2 * H * dim + H * vdim, decay, gain, 1e-5, 1.0, state, step, H, dim, vdim, out)
    a, b, sa, sb = _both(lens, 2 * H * dim + 2 * H * vdim, H * dim * vdim, H * vdim, run)
    _close(a, b, TOL)
    _close(sa, sb, TOL)


@pytest.mark.gpu
@pytest.mark.parametrize("H,dim,vdim", SHAPES)
@pytest.mark.parametrize("lens", LENS)
def test_exponential_gates(H, dim, vdim, lens, chunks):
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


@pytest.mark.gpu
@pytest.mark.parametrize("lens", LENS)
def test_state_space_groups(lens, chunks):
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


@pytest.mark.gpu
def test_a_value_that_is_not_a_number_reaches_no_earlier_token(chunks):
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


# ------------------------------------------------------------------ the same against the recurrences in 64 bits
def _walk64(q, k, v, decay, S):
    """q, k [n, H, dim], v [n, H, vdim], decay [n, H], S [H, vdim, dim]; outputs [n, H, vdim] and the state behind them."""
    out = []
    for t in range(len(q)):
        S = decay[t, :, None, None] * S + v[t, :, :, None] * k[t, :, None, :]
        out.append((S * q[t, :, None, :]).sum(-1))
    return torch.stack(out), S


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _against64(lens, width, n_state, inner, run, oracle, tol_out, taken):
    """`oracle(rows, state) -> (out, state)` of one sequence, in 64 bits."""
    g = torch.Generator().manual_seed(sum(lens) * 17 + width)
    rows = [torch.randn(n, width, generator=g) for n in lens]
    start = torch.rand(6, n_state, generator=g) * 0.5
    state, out = start.to(DEV), torch.full((sum(lens), inner), float("nan"), device=DEV)
    run(torch.cat(rows).to(DEV), state, _step(lens), out)
    want = [oracle(r.double(), start[SLOTS[i]].double()) for i, r in enumerate(rows)]
    _close(out.cpu(), torch.cat([w[0] for w in want]), tol_out)
    for i, w in enumerate(want):
        _close(state[SLOTS[i]].cpu(), w[1], TOL)
    assert torch.equal(state[[1, 3, 5]].cpu(), start[[1, 3, 5]]) and taken


@pytest.mark.gpu
@pytest.mark.parametrize("H,dim,vdim", SHAPES)
@pytest.mark.parametrize("lens", [[1, 1, 1], [65, 1, 34], [191, 200, 2]])
def test_constant_decay_in_64_bits(H, dim, vdim, lens, chunks):
    decay = torch.tensor([0.3, 0.995, 0.9, 1.0, 0.6, 0.05][:H])
    gain = torch.linspace(0.5, 1.5, H * vdim)

    def run(x, state, step, out):
        kernels.decay_attention(x, 0, 2 * H * dim + H * vdim, decay.to(DEV), gain.to(DEV), 1e-5, 1.3, state, step, H, dim, vdim, out)

    def oracle(x, S):
        n, silu = len(x), torch.nn.functional.silu
        q, k = (silu(x[:, c:c + H * dim]).view(n, H, dim) for c in (0, H * dim))
        v = silu(x[:, 2 * H * dim:2 * H * dim + H * vdim]).view(n, H, vdim)
        o, S = _walk64(q, k, v, decay.double().expand(n, H), S.view(H, vdim, dim))
        return _unit(o.reshape(n, -1), 1e-5) * gain.double() * torch.sigmoid(x[:, 2 * H * dim + H * vdim:]) * 1.3, S.reshape(-1)
    _against64(lens, 2 * H * dim + 2 * H * vdim, H * dim * vdim, H * vdim, run, oracle, TOL, chunks(lens))


@pytest.mark.gpu
@pytest.mark.parametrize("H,dim,vdim", SHAPES)
@pytest.mark.parametrize("lens", [[1, 1, 1], [65, 1, 34], [191, 200, 2]])
def test_exponential_gates_in_64_bits(H, dim, vdim, lens, chunks):
    bias, gain, cap = torch.randn(2, H, generator=torch.Generator().manual_seed(3)), torch.linspace(0.5, 1.5, H * vdim), 12.0
    cols, c = [], 0
    for size in (H * dim, H * dim, H * vdim, H * vdim, H, H):
        cols.append(c)
        c += size

    def run(x, state, step, out):
        b = bias.to(DEV)
        kernels.matrix_memory(x, *cols, b[0], b[1], cap, gain.to(DEV), 1e-5, state, step, H, dim, vdim, out)

    def oracle(x, state):
        n = len(x)
        q, k = (x[:, a:a + H * dim].view(n, H, dim) for a in cols[:2])
        v, g = (x[:, a:a + H * vdim] for a in cols[2:4])
        gi, gf = (cap * torch.tanh((x[:, a:a + H] + b.double()) / cap) for a, b in zip(cols[4:], bias))
        gf = torch.nn.functional.logsigmoid(gf)
        m, keep, take, tops = state[H * dim * (vdim + 1):], [], [], []
        for t in range(n):
            new = torch.maximum(gf[t] + m, gi[t])
            keep.append(torch.exp(gf[t] + m - new))
            take.append(torch.exp(gi[t] - new))
            tops.append(new)
            m = new
        v1 = torch.cat([v.view(n, H, vdim), torch.ones(n, H, 1, dtype=v.dtype)], -1) * torch.stack(take)[..., None]
        o, S = _walk64(q * dim ** -0.5, k, v1, torch.stack(keep), state[:H * dim * (vdim + 1)].view(H, vdim + 1, dim))
        o = o[..., :vdim] / (torch.maximum(o[..., vdim].abs(), torch.exp(-torch.stack(tops))) + 1e-6)[..., None]
        return _unit(o, 1e-5).reshape(n, -1) * gain.double() * torch.sigmoid(g), torch.cat([S.reshape(-1), m])
    _against64(lens, c, H * dim * (vdim + 1) + H, H * vdim, run, oracle, 1e-4, chunks(lens))


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[1, 1, 1], [65, 1, 34], [191, 200, 2]])
def test_state_space_in_64_bits(lens, chunks):
    H, G, N, vdim = 6, 2, 72, 48
    inner = H * vdim
    vec, gain = torch.randn(3, H, generator=torch.Generator().manual_seed(4)), torch.linspace(0.5, 1.5, inner)

    def run(x, state, step, out):
        proj, xbc, w = x[:, :inner + H].contiguous(), x[:, inner + H:].contiguous(), vec.to(DEV)
        kernels.state_space(proj, 0, inner, xbc, inner, inner + G * N, w[0], w[1], w[2], gain.to(DEV), 1e-5, 2, state, step, H, G, N, vdim, out)

    def oracle(x, S):
        n, w = len(x), vec.double()
        z, dt, xs = x[:, :inner], torch.nn.functional.softplus(x[:, inner:inner + H] + w[0]), x[:, inner + H:2 * inner + H].view(n, H, vdim)
        B, C = (x[:, a:a + G * N].view(n, G, N).repeat_interleave(H // G, 1) for a in (2 * inner + H, 2 * inner + H + G * N))
        o, S = _walk64(C, B, dt[..., None] * xs, torch.exp(-torch.exp(w[1]) * dt), S.view(H, vdim, N))
        y = (o + w[2][:, None] * xs).reshape(n, -1) * torch.nn.functional.silu(z)
        return _unit(y.view(n, 2, -1), 1e-5).reshape(n, -1) * gain.double(), S.reshape(-1)
    _against64(lens, 2 * inner + H + 2 * G * N, inner * N, inner, run, oracle, TOL, chunks(lens))
