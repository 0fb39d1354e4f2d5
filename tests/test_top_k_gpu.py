"""Top-k sampling (csrc/sampling.cu) where its candidates are few, many and tied, against a sort of the row."""
import pytest
import torch

from mini_llama_cpp_release_b200 import kernels
from mini_llama_cpp_release_b200.sampling import DeviceSampler, SamplingParams

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("vocab", [2, 37, 1000, 1024, 1028, 4099, 20480, 151936])
@pytest.mark.parametrize("k", [2, 40, 300, 1024])
@pytest.mark.parametrize("kind", ["normal", "rounded", "equal", "ascending", "one_share"])
def test_pick_lies_where_the_sorted_row_has_it(vocab, k, kind):
    g = torch.Generator().manual_seed(vocab + k)
    rows = torch.randn(5, vocab, generator=g)
    if kind == "rounded":
        rows = (rows * 2).round() / 2                # a hundred ids of a value: ties at the threshold
    elif kind == "equal":
        rows = torch.zeros(5, vocab)
    elif kind == "ascending":
        rows = torch.arange(vocab).float().expand(5, vocab).contiguous() / vocab
    elif kind == "one_share":
        rows[:, : min(vocab, 4000):4] += 30.0         # the largest in few threads' shares
    _check(rows, k)


def _check(rows, k):
    ids, pos = list(range(5)), [3, 9, 27, 81, 243]
    sampler = DeviceSampler(SamplingParams(0.7, k, 11), torch.device(DEV))
    got = sampler.sample(rows.to(DEV), ids, pos)
    kk = min(k, rows.shape[1])
    for b in range(5):
        # larger first, lower ids first among equal ones
        order = torch.argsort(rows[b].double(), descending=True, stable=True)[:kk]
        w = torch.exp((rows[b][order].double() - rows[b][order[0]].double()) / 0.7)
        cum = torch.cumsum(w, 0) / w.sum()
        at = (order == got[b]).nonzero()
        assert at.numel() == 1, (b, got[b])
        i = int(at)
        r = kernels.uniform_of(11, ids[b], pos[b])
        # a float32 running sum of up to 1,024 weights
        assert (cum[i - 1] if i else 0.0) <= r + 1e-4 and cum[i] >= r - 1e-4, (b, i, r)


@pytest.mark.parametrize("vocab,k", [(2047, 127), (2048, 128), (2048, 129), (4096, 256), (4097, 257), (12800, 800), (12816, 801), (40000, 800)])
@pytest.mark.parametrize("kind", ["normal", "masked", "few_kept"])
def test_both_ways_of_finding_the_largest_at_the_lines_between_them(vocab, k, kind):
    """Two reads up to a sixteenth of the row and 800, from 2,048 logits on; the digits elsewhere, and where one value fills the row."""
    g = torch.Generator().manual_seed(vocab * 3 + k)
    rows = torch.randn(5, vocab, generator=g)
    if kind == "masked":
        rows[:, torch.randperm(vocab, generator=g)[: vocab - 2 * k]] = float("-inf")
    elif kind == "few_kept":
        rows[:, torch.randperm(vocab, generator=g)[: vocab - k // 2]] = torch.finfo(torch.float32).min
    _check(rows, k)
