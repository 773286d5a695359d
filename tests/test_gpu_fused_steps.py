"""Steps in which sublayers add to the residual stream at their last product's store, or form the norm in front of them inside their first
product, against the same steps with neither (a step whose intermediates are tapped takes every kernel by itself): the same bits, in
the logits, the keys and values and the states, launch by launch and captured."""
import sys
from collections import Counter

import pytest
import torch

pytestmark = pytest.mark.gpu

# wide enough that the streaming product has a strip for every SM; dense and routed feed-forwards after both kinds of mixer
CONFIG = {"architectures": ["Lfm2MoeForCausalLM"], "vocab_size": 512, "hidden_size": 2048, "num_hidden_layers": 5,
          "layer_types": ["conv", "full_attention", "conv", "full_attention", "conv"], "num_attention_heads": 32,
          "num_key_value_heads": 8, "conv_L_cache": 3, "conv_bias": False, "num_dense_layers": 3, "intermediate_size": 1536,
          "num_experts": 8, "num_experts_per_tok": 2, "moe_intermediate_size": 256, "norm_topk_prob": True, "use_expert_bias": True,
          "routed_scaling_factor": 1.0, "rope_theta": 1e6, "norm_eps": 1e-5, "tie_word_embeddings": True, "max_position_embeddings": 4096}
PAGE = 16


@pytest.fixture(scope="module")
def model():
    from snowllm_b200.loader import build_model
    from snowllm_b200.weights import random_tensors
    from snowllm_b200.weights.loader import load_tensors
    model = build_model(CONFIG, "bfloat16")
    tensors = random_tensors(model, 3, torch.bfloat16, fan_in_scaled=True, norm_jitter=0.1)
    load_tensors(model, {k: v.cuda() for k, v in tensors.items()}, "cuda")
    return model


@pytest.fixture
def called(monkeypatch):
    """How often a norm was formed in a product, a convolution run at a product's store, a product added to the stream."""
    from snowllm_b200.ops import kernels
    calls = Counter()

    def count(owner, name):
        f = getattr(owner, name)
        monkeypatch.setattr(owner, name, lambda *a, **kw: calls.update([name]) or f(*a, **kw))
    count(kernels.PendingNorm, "product")
    count(kernels, "conv_step")
    count(sys.modules["snowllm_b200.ops.linear"], "linear_add")
    return calls


def sides(model, requests, graphs=False):
    from snowllm_b200.cache import CacheManager
    from snowllm_b200.engine import ModelRunner
    out = []
    for tapped in (False, True):
        cache = CacheManager(model.cache_specs(), PAGE, 16 * requests, requests, model.dtype, "cuda")
        for t in (*cache.paged_tensors(), *cache.state_tensors()):
            t.zero_()
        runner = ModelRunner(model, cache, "cuda", use_graphs=graphs and not tapped)
        out.append((runner, cache, [cache.admit() for _ in range(requests)], tapped))
    return out


def step(side, tokens):
    """The step's logits, of every last token."""
    from snowllm_b200.engine import StepEntry
    runner, cache, held, tapped = side
    for rc, t in zip(held, tokens):
        assert cache.ensure(rc, rc.num_tokens + len(t))
    runner.taps = [] if tapped else None
    return runner.step([StepEntry(rc, t, [len(t) - 1]) for rc, t in zip(held, tokens)]).clone()


def same(a, b):
    for x, y in zip((*a[1].paged_tensors(), *(t[:len(a[2])] for t in a[1].state_tensors())),
                    (*b[1].paged_tensors(), *(t[:len(b[2])] for t in b[1].state_tensors()))):
        assert torch.equal(x, y)


def draw(gen, *lengths):
    return [torch.randint(0, CONFIG["vocab_size"], (n,), generator=gen).tolist() for n in lengths]


# one row over, one at the line of the tensor-core products (17 rows), two requests' portions of one step
@pytest.mark.parametrize("lengths", [(16,), (17,), (40,), (23, 150)])
def test_prompts(model, called, lengths):
    fused, plain = sides(model, len(lengths))
    gen = torch.Generator().manual_seed(sum(lengths))
    for _ in range(2):                                    # a fresh portion, and one that goes on
        tokens = draw(gen, *lengths)
        called.clear()
        a = step(fused, tokens)
        # five mixers, three dense feed-forwards
        assert called == ({"linear_add": 8} if sum(lengths) > 16 else {})
        called.clear()
        b = step(plain, tokens)
        assert not called
        assert torch.equal(a, b) and a.isfinite().all()
        same(fused, plain)


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("requests", [1, 2, 3])
def test_one_token_steps(model, called, requests, graphs):
    fused, plain = sides(model, requests, graphs)
    gen = torch.Generator().manual_seed(requests)
    first = draw(gen, *(40 + 7 * i for i in range(requests)))
    step(fused, first), step(plain, first)
    for i in range(30):                                   # over a page's edge, and over a capture's (64 positions)
        tokens = draw(gen, *[1] * requests)
        called.clear()
        a = step(fused, tokens)
        if not graphs or i == 0:                          # (a captured step calls them while it is captured)
            assert (called["product"] >= 5 and called["conv_step"] >= 3) if requests <= 2 else not called, called
        called.clear()
        b = step(plain, tokens)
        assert not called["product"] and torch.equal(a, b) and a.isfinite().all(), i
        same(fused, plain)
    assert fused[0].graph_replays == (30 if graphs else 0)


def test_rows_do_not_depend_on_how_many_there_are(model):
    """The same request alone, with a second one and with a third: one row forms its norms inside its products, two rows do, and
    three rows have kernels for them."""
    gen = torch.Generator().manual_seed(9)
    prompts, follow = draw(gen, 33, 50, 21), [draw(gen, 1, 1, 1) for _ in range(8)]
    outs = []
    for n in (1, 2, 3):
        side = sides(model, n)[0]
        for rc, t in zip(side[2], prompts):               # (each prompt in a step of its own)
            one = (side[0], side[1], [rc], False)
            step(one, [t])
        outs.append(torch.stack([step(side, tokens[:n])[0] for tokens in follow]))
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
