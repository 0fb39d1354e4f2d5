"""A sequence's single tokens are the same sum in float32 whatever else is in the batch."""
import pytest
import torch

import helpers
import mini_llama_cpp_release_b200 as ml
from types import SimpleNamespace
from mini_llama_cpp_release_b200.engine import MiniBatch
from mini_llama_cpp_release_b200.parts.attention import choose_splits


def test_the_keys_of_a_single_token_are_shared_out_by_its_own_length_alone():
    tile = 32                                            # csrc/attention_simt.cu: a split takes ceil(tiles / splits) tiles
    for length in [*range(1, 1300), 2047, 2048, 2049, 5000, 40000]:
        tiles = -(-length // tile)
        shares = set()
        for n_seqs in (1, 3, 24, 64, 1000):
            for most in (length, length + 1, 2 * length, 256, 1024, 65536):        # the longest of the batch, or the runner's
                if most >= length:
                    n = choose_splits(SimpleNamespace(max_q_len=1, n_seqs=n_seqs, max_kv_len=most), 14, 2, 148, 2)
                    shares.add(-(-tiles // n))
        assert len(shares) == 1, (length, shares)


@pytest.mark.gpu
def test_float32_logits_of_a_sequence_are_the_same_bits_in_any_batch():
    folder = helpers.model_folder("C", std=0.1)          # 14 heads on 2
    prompts = [helpers.random_tokens(1 + (37 * i) % 290, 777, 500 + i) for i in range(48)]
    fed = [helpers.random_tokens(6, 777, 900 + i) for i in range(48)]

    def run(which):
        ctx = ml.load(folder, dtype="float32", max_tokens=64 * 400, max_seqs=48).context
        slots = [ctx.acquire() for _ in which]
        for s, i in zip(slots, which):                   # (a norm of 256 rows and more sums a row in another order)
            ctx.forward_batch(MiniBatch.from_tokens(s, prompts[i], want=[]))
        return torch.stack([ctx.forward_batch(MiniBatch.decode(slots, [fed[i][t] for i in which])) for t in range(6)])
    whole = run(range(48))
    for which in ([47], [13], [0], list(range(24)), [5, 40]):
        assert torch.equal(run(which), whole[:, which]), which


@pytest.mark.gpu
def test_sampled_ids_of_a_request_are_the_same_in_any_batch():
    llm = helpers.engine(helpers.model_folder("C", std=0.1), "float32", 48 * 384)
    prompts = [helpers.random_tokens(1 + (53 * i) % 240, 777, 80 + i) for i in range(48)]
    together = llm.generate(prompts, n_predict=24, temperature=0.9, seed=77, stop_token_ids=[])
    for batch in (1, 5, 24):
        assert llm.generate(prompts, n_predict=24, temperature=0.9, seed=77, stop_token_ids=[], max_batch=batch) == together, batch
