"""What a serving engine refuses before any work is issued, and its small host-side pieces (CPU)."""
import gc
import weakref

import numpy as np
import pytest
import torch

from brain_b200.models.config import QwenConfig
from brain_b200.models.qwen3 import Qwen3
from brain_b200.serve.base import read_back
from brain_b200.serve.engine import QwenEngine


def _engine(**kw):
    cfg = QwenConfig(vocab=61, block_size=96, n_layers=1, d_model=32, n_heads=4, n_kv_heads=2, head_dim=8, d_ff=64)
    return QwenEngine(Qwen3(cfg).init_weights(1).eval(), block_size=8, num_blocks=16, max_seq_len=64, **kw)


@pytest.mark.parametrize("position,window", [(-1, 1), (64, 1), (63, 2), (1 << 30, 1)])
def test_positions_outside_the_block_table_are_refused(position, window, monkeypatch):
    """Before the step reaches the device: its kernels look up the table unchecked."""
    eng = _engine()
    reached = []
    monkeypatch.setattr(eng, "_decode_steps", lambda *a: reached.append(a))
    tables = np.arange(16, dtype=np.int32).reshape(2, 8)
    with pytest.raises(IndexError):
        eng.decode(np.array([1, 2], dtype=np.int32), np.array([3, position], dtype=np.int32), tables, window=window)
    assert not reached
    if window == 1:
        with pytest.raises(IndexError):
            eng.mixed_step([(np.array([5, 6], dtype=np.int32), 0, tables[0], True, True)], np.array([2], dtype=np.int32),
                           np.array([position], dtype=np.int32), tables[1:])
        with pytest.raises(IndexError):
            eng.prefill_chunk(np.array([5], dtype=np.int32), position, tables[0], True)
        with pytest.raises(IndexError):
            eng.prefill_batch([(np.array([5], dtype=np.int32), s, t, True, True) for s, t in zip((0, position), tables)])


def test_the_last_position_of_a_table_is_served():
    eng = _engine()
    tables = np.arange(8, dtype=np.int32)[None, :]
    toks, _ = eng.decode(np.array([1], dtype=np.int32), np.array([62], dtype=np.int32), tables, window=2)
    assert len(toks[0]) == 2


@pytest.mark.parametrize("shape", [(0,), (0, 2), (3,), (3, 1), (3, 4)])
def test_read_back_of_tokens_and_candidates(shape):
    g = torch.Generator().manual_seed(1)
    tokens = torch.randint(0, 1 << 30, shape, generator=g, dtype=torch.int32)
    ids = torch.randint(0, 1 << 30, (shape[0], 5), generator=g, dtype=torch.int32)
    logits = torch.randn(shape[0], 5, generator=g)
    picked, cands = read_back(tokens, (ids, logits))
    assert picked == tokens.tolist()
    assert cands == [list(zip(i, v)) for i, v in zip(ids.tolist(), logits.tolist())]
    assert read_back(tokens, None) == (tokens.tolist(), None)


def test_an_engine_goes_with_its_last_reference():
    """Also one with the native forward: what waits for a collection may be freed while another engine's step is captured."""
    from brain_b200.serve.native import NativeForward
    eng = _engine()
    eng.native = NativeForward(eng)
    gone = weakref.ref(eng)
    collecting = gc.isenabled()
    gc.disable()
    try:
        del eng
        assert gone() is None
    finally:
        if collecting:
            gc.enable()
