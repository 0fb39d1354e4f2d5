"""The page tables a captured decode step reads (engine/decode_runner.py): after every step they are the cache's page lists, row by row."""
import pytest
import torch

import helpers
from helpers import model_folder, random_tokens
from mini_llama_cpp_release_b200.engine import MiniBatch
from mini_llama_cpp_release_b200.engine.decode_runner import DecodeRunner
from mini_llama_cpp_release_b200.sampling import DeviceSampler, SamplingParams

pytestmark = pytest.mark.gpu


def test_every_row_of_the_tables_follows_the_cache(monkeypatch):
    """Five sequences in a batch of six rows (the last is repeated), one group that keeps all keys and one that keeps a window of
    24: rows gain pages at other steps than they lose them, some at the same step as another, the repeated row among them."""
    llm = helpers.ml.load(model_folder("W"), dtype="bfloat16", max_tokens=4096)
    ctx, cache = llm.context, llm.context.cache
    groups = range(len(cache.groups))
    assert len(cache.groups) == 2
    changes, before = [], {}

    def checked(runner):
        torch.cuda.synchronize()
        rows = runner._padded_slots
        assert len(rows) == runner.B == 6 and rows[4] == rows[5]
        changed = []
        for g in groups:
            table = runner.view(f"pages{g}").view(runner.B, runner.pages_per_seq).tolist()
            for b, slot in enumerate(rows):
                pages = cache.page_lists[slot][g]
                assert table[b] == pages + [-1] * (runner.pages_per_seq - len(pages)), (g, b)
                if before.get((g, b), pages) != pages:
                    changed.append((g, b))
                before[g, b] = list(pages)
        changes.append(changed)
        return replay(runner)

    replay = DecodeRunner.replay
    monkeypatch.setattr(DecodeRunner, "replay", checked)
    lengths = (40, 63, 1, 130, 17)                 # 63 leaves its window's first page behind as 40 gets its second
    prompts = [random_tokens(n, 301, n) for n in lengths]
    slots = [ctx.acquire() for _ in prompts]
    sampler = DeviceSampler(SamplingParams(), llm.model.runtime.device)
    tokens = ctx.forward_batch(MiniBatch.prefill(slots, prompts)).argmax(dim=1).tolist()
    for _ in range(130):
        tokens, _ = ctx.decode_and_sample(slots, tokens, sampler, list(range(5)))
    for s in slots:
        ctx.release(s)
    rows = [{b for _, b in c} for c in changes]
    assert any(len(r) == 1 for r in rows) and any({0, 1} <= r for r in rows) and any({4, 5} <= r for r in rows)
    assert any({g for g, _ in c} == {1} for c in changes)        # only the window's group: a page given back

