"""Which shapes of step get a captured graph, and that a captured step answers as an issued one does."""
import random

import pytest
import torch

import betepel_helpers
import helpers
import mepolix_helpers
import mini_llama_cpp_release_b200 as ml
from mini_llama_cpp_release_b200.engine import MiniBatch
from mini_llama_cpp_release_b200.engine.step_shapes import SHAPES_SEEN, StepShapes


class Book:
    """Sends shapes and counts captures."""

    def __init__(self, sights=2, places=3, idle=20):
        self.shapes, self.places, self.idle, self.captures = StepShapes(sights), places, idle, []

    def send(self, *keys):
        for key in keys:
            capture, leaving = self.shapes.coming(key, self.places, self.idle)
            assert not (capture and key in self.shapes.kept)
            if capture:
                self.shapes.keep(key, leaving)
                self.captures.append(key)
            assert len(self.shapes.kept) <= self.places
        return self

    @property
    def kept(self):
        return set(self.shapes.kept)


def test_a_shape_is_captured_at_its_sight():
    assert Book(2).send("a").kept == set() and Book(2).send("a", "b", "a").kept == {"a"}
    assert Book(8).send(*"aaaaaaa").kept == set() and Book(8).send(*"aaaaaaaa").kept == {"a"}
    assert Book(2, places=0).send(*"aaaa").kept == set()


def test_more_shapes_in_turn_than_places_are_not_captured_over_and_over():
    b = Book(places=3, idle=20)
    for _ in range(50):
        b.send(*"abcdefgh")
    assert len(b.captures) == 3
    b = Book(places=8, idle=64)                      # in any order
    rng = random.Random(1)
    for _ in range(100):
        b.send(*rng.sample(range(16), 16))
    assert len(b.captures) == 8


def test_a_frequent_shape_takes_the_place_of_a_rare_one():
    b = Book(places=3, idle=1000).send(*"aabbcc")
    for i in range(30):                              # each of the three comes at every sixth step, the new one at every second
        b.send("x", "abc"[i % 3])
    assert "x" in b.kept and len(b.captures) == 4
    b = Book(places=3, idle=1000).send(*"aabbcc")
    for i in range(60):                              # as rare as they are: no change
        b.send(*"abcx")
    assert b.kept == set("abc")


def test_a_place_that_nobody_uses_goes_to_the_next_that_comes_again():
    b = Book(places=2, idle=10).send(*"aabb")
    b.send(*"bbbbbb").send("x", "x")
    assert b.kept == {"a", "b"}                      # a: ten steps ago
    b.send("x")
    assert b.kept == {"b", "x"}


def test_a_failed_capture_leaves_the_book_as_it_was():
    s = StepShapes(2)
    s.coming("a", 1, 10)
    assert s.coming("a", 1, 10) == (True, None) and s.coming("a", 1, 10) == (True, None)
    s.keep("a", None)
    assert s.coming("a", 1, 10) == (False, None)


def test_shapes_without_a_place_are_forgotten_in_the_order_of_their_last_coming():
    b = Book(2).send("a").send(*range(SHAPES_SEEN - 1)).send("a")
    assert "a" in b.kept
    b = Book(2).send("a").send(*range(SHAPES_SEEN)).send("a")
    assert "a" not in b.kept


def _rounds(ctx, vocab, lens, n_rounds, fresh):
    """`n_rounds` steps of one shape, each with other tokens in slots of their own, and a decoded token behind each."""
    for r in range(n_rounds):
        seqs = [helpers.random_tokens(n, vocab, 100 * r + n) for n in lens]
        answers = []
        for c in (ctx, fresh):
            hold = [c.acquire() for _ in range(r % 3)]                 # other slots than the round before
            slots = [c.acquire() for _ in seqs]
            got = c.forward_batch(MiniBatch.prefill(slots, seqs))
            answers.append(torch.cat([got, c.forward_batch(MiniBatch.decode(slots, [3 + i for i in range(len(lens))]))]))
            for s in slots + hold:
                c.release(s)
        yield answers


# The captured step runs the kernels of the issued one: in float32 the same bits; in bfloat16 the order of a few atomic adds
# differs, which these models magnify as much as any other rounding (the bounds of their own tests)
MODELS = {"attention": (lambda: helpers.model_folder("C"), helpers.TOL["bfloat16"]),
          "delta rule, recurrence": (lambda: mepolix_helpers.folder_of("mixed"), mepolix_helpers.TOL["bfloat16"]),
          "matrix memory, experts": (lambda: betepel_helpers.folder_of("mixed"), betepel_helpers.TOL["bfloat16"][0])}


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [(23,), (9, 14, 1)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("model", list(MODELS))
def test_short_steps_are_captured_at_their_eighth_coming_and_answer_alike(model, dtype, lens):
    folder, tol = MODELS[model][0](), MODELS[model][1]
    ctx, issued = (ml.load(folder, dtype=dtype, max_tokens=2048, max_seqs=8).context for _ in range(2))
    assert ctx.use_graphs
    issued.use_graphs = False
    vocab = ctx.model.config.vocab_size
    for r, (got, ref) in enumerate(_rounds(ctx, vocab, lens, 11, issued)):
        assert torch.equal(got, ref) if dtype == "float32" else helpers.rel_err(got, ref) <= tol, r
        keys = [k for k in ctx.__dict__.get("_step_graphs", {}) if k[0] == sum(lens)]
        assert len(keys) == (1 if r >= 7 else 0), r
    ctx.cache.check()


@pytest.mark.gpu
def test_places_of_a_context_are_kept_refused_and_given_up():
    ctx = ml.load(helpers.model_folder("A"), dtype="float32", max_tokens=4096).context
    ctx.STEP_GRAPHS, ctx.STEP_GRAPH_IDLE = 2, 3

    def send(n):
        s = ctx.acquire()
        out = ctx.forward_batch(MiniBatch.from_tokens(s, [i % 512 for i in range(n)]))
        ctx.release(s)
        return out.clone()

    def kept():
        return sorted(k[0] for k in ctx._step_graphs)
    first = {n: send(n) for n in (70, 80, 90)}
    for n in (70, 80):
        send(n)
    assert kept() == [70, 80]
    assert torch.equal(send(90), first[90]) and kept() == [70, 80]          # no place
    for n in range(1, 40):                                                  # short steps take none of the long ones' places
        send(n)
    assert kept() == [70, 80]
    for _ in range(3):
        assert torch.equal(send(80), first[80])
    assert torch.equal(send(90), first[90]) and kept() == [80, 90]          # 70 was not used for more than three long steps
    for n in (70, 80, 90):
        assert torch.equal(send(n), first[n])


@pytest.mark.gpu
def test_a_long_prompt_is_replayed_however_many_single_tokens_lie_between():
    ctx = ml.load(helpers.model_folder("A"), dtype="float32", max_tokens=4096).context
    for r in range(2):
        s = ctx.acquire()
        ctx.forward_batch(MiniBatch.from_tokens(s, [i % 512 for i in range(100)]))
        for i in range(90):
            ctx.forward_batch(MiniBatch.single(s, i))
        ctx.release(s)
    assert [k[0] for k in ctx._step_graphs] == [100]


@pytest.mark.gpu
def test_steps_above_the_longest_that_is_captured_are_issued():
    ctx = ml.load(helpers.model_folder("A"), dtype="float32", max_tokens=4096).context
    ctx.STEP_GRAPH_MAX_TOKENS = 120
    outs = []
    for _ in range(3):
        for n in (120, 121):
            s = ctx.acquire()
            outs.append(ctx.forward_batch(MiniBatch.from_tokens(s, [i % 512 for i in range(n)])).clone())
            ctx.release(s)
    assert [k[0] for k in ctx._step_graphs] == [120]
    assert all(torch.equal(outs[i], outs[i % 2]) for i in range(6))
