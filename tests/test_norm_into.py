"""A norm is left to the product that reads it only where both run the library's own `forward`."""
from types import SimpleNamespace

import pytest
import torch

import helpers
import mini_llama_cpp_release_b200 as ml
from mini_llama_cpp_release_b200.config import ModelConfig, ModelSpec, PartSpec, prenorm_layer, sequential_schedule
from mini_llama_cpp_release_b200.engine import MiniBatch
from mini_llama_cpp_release_b200.models.qwen2 import LAYER_NAMES
from mini_llama_cpp_release_b200.parts.attention import GQAttention
from mini_llama_cpp_release_b200.parts.block import norm_into
from mini_llama_cpp_release_b200.parts.embedding import LinearHead
from mini_llama_cpp_release_b200.parts.feed_forward import SwiGLU
from mini_llama_cpp_release_b200.parts.linear import Linear
from mini_llama_cpp_release_b200.parts.norm import NormedStream, RMSNorm


@ml.register_part("norm", "toy_folded_norm")
class FoldedNorm(RMSNorm):
    """The RMS norm with its negative entries halved: no gain makes it a plain one."""

    def forward(self, x, delta=None, out_dtype=None):
        h = super().forward(x, delta, out_dtype)
        return torch.where(h < 0, h * 0.5, h)


def _bound(part, **tensors):
    rt = SimpleNamespace(dtype=torch.bfloat16, device=torch.device("cpu"), n_sms=148)
    part.bind(lambda name: tensors[name], rt)
    return part


def _norm(cls=RMSNorm):
    return _bound(cls("n.", 128, 1e-6), **{"n.weight": torch.ones(128)})


TAKES = SimpleNamespace(takes_normed_stream=lambda n: True)


def test_the_plain_norm_is_left_to_a_reader_that_takes_it():
    x = torch.randn(4, 128)
    h = norm_into(_norm(), TAKES, x, None)
    assert isinstance(h, NormedStream) and h.x is x


def test_another_forward_is_called(monkeypatch):
    x, marker = torch.randn(4, 128), torch.zeros(1)

    class Own(RMSNorm):
        def forward(self, x, delta=None, out_dtype=None):
            return marker
    assert norm_into(_norm(Own), TAKES, x, None, 4) is marker

    class OwnBelow(Own):
        pass
    assert norm_into(_norm(OwnBelow), TAKES, x, None, 4) is marker
    wrapped = _norm()
    wrapped.forward = lambda *a, **k: marker
    assert norm_into(wrapped, TAKES, x, None, 4) is marker
    plain = _norm()
    monkeypatch.setattr(RMSNorm, "forward", lambda self, *a, **k: marker)
    assert norm_into(plain, TAKES, x, None, 4) is marker


def _readers():
    w = torch.zeros(128, 128, dtype=torch.bfloat16)
    head = LinearHead("h.", 128, 128)
    ffn = SwiGLU("f.", 128, 128)
    att = GQAttention("a.", hidden_size=128, num_heads=4, num_kv_heads=2, head_dim=32, qkv_bias=False,
                      position=PartSpec("position", "rope_neox", dict(head_dim=32, theta=1e4, max_positions=64)))
    _bound(head, **{n.name: w for n in head.all_tensors()})
    _bound(ffn, **{n.name: w for n in ffn.all_tensors()})
    _bound(att, **{n.name: torch.zeros(n.shape, dtype=torch.bfloat16) for n in att.all_tensors()})
    return head, ffn, att


def test_a_reader_with_another_forward_is_given_rows(monkeypatch):
    readers = _readers()
    assert all(r.takes_normed_stream(4) for r in readers)
    for r in readers:
        r.forward = lambda *a, **k: None
        assert not r.takes_normed_stream(4)
        del r.forward
        monkeypatch.setattr(type(r), "forward", lambda self, *a, **k: None)
        assert not r.takes_normed_stream(4)
        monkeypatch.undo()
        assert r.takes_normed_stream(4)


def test_a_head_with_another_product_is_given_rows():
    class Scaled(Linear):
        def __call__(self, x, out_dtype=torch.float32, partial_ok=False):
            return super().__call__(x, out_dtype, partial_ok) * 2
    head = _readers()[0]
    head.proj = Scaled(head.proj.weight, head.proj.runtime)
    assert not head.takes_normed_stream(4)
    head.proj = lambda x, out_dtype: x                   # no `Linear` at all
    assert not head.takes_normed_stream(4)


@ml.register_architecture("ToyFoldedNormLM")
def folded_norm_lm(c: ModelConfig) -> ModelSpec:
    norm = PartSpec("norm", "toy_folded_norm", dict(size=c.hidden_size, eps=1e-5))
    rope = PartSpec("position", "rope_neox", dict(head_dim=c.head_dim, theta=1e4, max_positions=256))
    att = PartSpec("mixer", "gqa_attention", dict(hidden_size=c.hidden_size, num_heads=c.num_attention_heads,
                                                  num_kv_heads=c.num_key_value_heads, head_dim=c.head_dim, qkv_bias=False, position=rope))
    ffn = PartSpec("feed_forward", "swiglu", dict(hidden_size=c.hidden_size, intermediate_size=c.intermediate_size))
    layers = tuple(prenorm_layer(f"model.layers.{i}.", att, ffn, norm, norm, LAYER_NAMES) for i in range(2))
    return ModelSpec(c, PartSpec("embedding", "token_embedding", dict(vocab_size=c.vocab_size, hidden_size=c.hidden_size)),
                     layers, sequential_schedule(len(layers)), norm,
                     PartSpec("head", "linear_head", dict(vocab_size=c.vocab_size, hidden_size=c.hidden_size)))


@pytest.mark.gpu
def test_a_norm_of_its_own_answers_alike_in_prompts_and_in_small_steps(tmp_path):
    raw = dict(architectures=["ToyFoldedNormLM"], hidden_size=128, intermediate_size=192, num_hidden_layers=2, num_attention_heads=4,
               num_key_value_heads=2, head_dim=32, vocab_size=160, max_position_embeddings=256, rope_theta=1e4, rms_norm_eps=1e-5)
    folder = ml.write_random_model(ModelConfig.from_dict(raw), str(tmp_path / "folded"), 3, std=0.1)
    tokens = helpers.random_tokens(100, 160, 5)
    ctx = ml.load(folder, dtype="float32", max_tokens=512).context
    ref = ctx.forward_batch(MiniBatch.from_tokens(ctx.acquire(), tokens, want=list(range(100))))
    ctx = ml.load(folder, dtype="bfloat16", max_tokens=512).context
    whole = ctx.forward_batch(MiniBatch.from_tokens(ctx.acquire(), tokens, want=list(range(100))))
    slot, rows, at = ctx.acquire(), [], 0
    for n in (1, 8, 3, 16, 12):
        rows.append(ctx.forward_batch(MiniBatch.from_tokens(slot, tokens[at:at + n], want=list(range(n)))))
        at += n
    assert helpers.rel_err(whole, ref) <= helpers.TOL["bfloat16"]
    assert helpers.rel_err(torch.cat(rows), ref[:at]) <= helpers.TOL["bfloat16"]
