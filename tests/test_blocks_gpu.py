"""A block as one autograd node against the same block operator by operator."""
import pytest
import torch

from brain_b200.engine import Trainer
from brain_b200.models import gpt2, qwen3
from brain_b200.models.config import GptConfig, QwenConfig
from brain_b200.ops.blocks import fused_ok

pytestmark = pytest.mark.gpu


def _qwen(bias, norm):
    return qwen3.Qwen3(QwenConfig(vocab=160, block_size=96, n_layers=3, d_model=192, n_heads=3, n_kv_heads=1, head_dim=64, d_ff=328,
                                  attn_bias=bias, qk_norm=norm)).init_weights(seed=1)


MODELS = {"qwen": lambda: _qwen(False, True), "qwen-bias": lambda: _qwen(True, False),
          "gpt": lambda: gpt2.Gpt2(GptConfig(vocab=160, block_size=96, n_layers=3, d_model=192, n_heads=3, d_ff=328)).init_weights(seed=1)}


@pytest.mark.parametrize("rows", [1, 3])
@pytest.mark.parametrize("name", list(MODELS))
def test_gradients_are_those_of_the_operators(name, rows, monkeypatch):
    g = torch.Generator().manual_seed(rows)
    ids = torch.randint(0, 160, (rows, 78), generator=g, dtype=torch.int32)
    runs = []
    for fused in (True, False):
        if not fused:
            monkeypatch.setattr(qwen3, "fused_ok", lambda *a: False)
            monkeypatch.setattr(gpt2, "fused_ok", lambda *a: False)
        tr = Trainer(MODELS[name](), device=torch.device("cuda:0"))
        tr.zero_grads()
        loss = tr.forward_backward(ids[:, :-1].contiguous(), ids[:, 1:].contiguous(), rows, 1.0 / (77 * rows))
        runs.append((float(loss), tr.store.grads.double().clone()))
    (l0, g0), (l1, g1) = runs
    assert l0 == l1                                    # the forward launches are the same
    # the residual gradients are summed before a rounding to bf16 instead of after one: 2^-9 of a value a block, three blocks
    assert float((g0 - g1).norm() / g1.norm()) < 3 * 3 * 2 ** -9


def _wide(name):
    if name == "gpt":
        return gpt2.Gpt2(GptConfig(vocab=160, block_size=320, n_layers=2, d_model=256, n_heads=2, d_ff=328)).init_weights(seed=2)
    return qwen3.Qwen3(QwenConfig(vocab=160, block_size=320, n_layers=2, d_model=256, n_heads=4, n_kv_heads=2, head_dim=128, d_ff=328)).init_weights(seed=2)


@pytest.mark.parametrize("name", ["qwen", "gpt"])
def test_wide_heads_many_rows_and_two_micro_batches(name, monkeypatch):
    """128-wide heads, 300 rows a micro-batch (products on other forms than those of few rows), gradients of two micro-batches
    added up, and every parameter reported once a micro-batch, behind its gradient."""
    from brain_b200.ops import functional as F
    g = torch.Generator().manual_seed(3)
    ids = torch.randint(0, 160, (2, 301), generator=g, dtype=torch.int32)
    runs = []
    for fused in (True, False):
        if not fused:
            monkeypatch.setattr(qwen3, "fused_ok", lambda *a: False)
            monkeypatch.setattr(gpt2, "fused_ok", lambda *a: False)
        model = _wide(name)
        tr = Trainer(model, device=torch.device("cuda:0"))
        tr.zero_grads()
        told = []
        monkeypatch.setattr(F, "grad_ready_hook", lambda p: told.append((id(p), float(p.main_grad.abs().sum()))))
        loss = tr.forward_backward(ids[:, :-1].contiguous(), ids[:, 1:].contiguous(), 1, 1.0 / 600)
        monkeypatch.setattr(F, "grad_ready_hook", None)
        block = {id(p) for b in model.blocks for p in b.parameters()}
        seen = [i for i, _ in told if i in block]
        assert len(seen) == 2 * len(block) and set(seen) == block
        assert all(v > 0 for i, v in told if i in block)
        last = {i: v for i, v in told}                  # what a parameter's last report saw is its final gradient
        assert all(last[id(p)] == float(p.main_grad.abs().sum()) for b in model.blocks for p in b.parameters())
        runs.append((float(loss), tr.store.grads.double().clone()))
    (l0, g0), (l1, g1) = runs
    assert l0 == l1
    assert float((g0 - g1).norm() / g1.norm()) < 2 * 3 * 2 ** -9      # as above, two blocks


def test_frozen_parameters_and_saved_tensor_hooks(monkeypatch):
    """A block with a frozen weight runs operator by operator: the weight gets no gradient, all others those of a model that
    runs so throughout; and hooks on saved tensors see a block's activations."""
    ids = torch.randint(0, 160, (2, 78), generator=torch.Generator().manual_seed(4), dtype=torch.int32)
    runs = []
    for fused in (True, False):
        took = []
        for mod in (qwen3, gpt2):
            monkeypatch.setattr(mod, "fused_ok", lambda x, params, f=fused: took.append(f and fused_ok(x, params)) or took[-1])
        model = MODELS["qwen"]()
        frozen = model.blocks[1].wo.requires_grad_(False)
        tr = Trainer(model, device=torch.device("cuda:0"))
        seen = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t.shape) or t, lambda t: t):
            tr.zero_grads()
            tr.forward_backward(ids[:, :-1].contiguous(), ids[:, 1:].contiguous(), 2, 1e-2)
        assert took == ([True, False, True] if fused else [False] * 3)
        assert (154, 328) in seen                          # the feed-forward activation
        assert frozen.grad is None and (getattr(frozen, "main_grad", None) is None or not bool((frozen.main_grad != 0).any()))
        runs.append(tr.store.grads.double().clone())
    assert bool((model.blocks[0].wo.main_grad != 0).any())
    assert float((runs[0] - runs[1]).norm() / runs[1].norm()) < 3 * 3 * 2 ** -9
