"""What decides whether a captured step may stand in for the step, and what the capture holds on to.  Nothing is captured
here: the engine runs on the CPU with the attention whose state a capture bakes in."""
import copy
import gc
import weakref

import pytest
import torch

from torchft_b200.models.llama import LLAMA_TINY, Tcgen05Attention
from torchft_b200.parallel.hsdp import ShardedLlamaTrainer, _StepGraph

B, S = 1, 16


def _trainer(cls=ShardedLlamaTrainer):
    cfg = copy.copy(LLAMA_TINY)
    return cls(cfg, B, S, torch.device("cpu"), attention=Tcgen05Attention(cfg), logit_chunks=2)


def _batch(tr, seed=0):
    return torch.randint(0, tr.cfg.vocab_size, (2, B, S), generator=torch.Generator().manual_seed(seed))


def test_log_sum_exps_stay_where_they_are():
    tr = _trainer()
    tok, tgt = _batch(tr)
    tr.engine.forward(tok, tgt)
    first = {layer: weakref.ref(lse) for layer, (_, _, lse) in tr.engine.attn._saved.items()}
    assert len(first) == tr.cfg.n_layers
    tr.engine.backward(tok)
    for _ in range(3):  # no backward pass
        tr.engine.forward(tok, tgt)
        gc.collect()
        assert all(ref() is not None for ref in first.values())
        assert {layer: id(lse) for layer, (_, _, lse) in tr.engine.attn._saved.items()} == {k: id(ref()) for k, ref in first.items()}


def test_passes_without_a_backward_replace_no_tensor():
    """Loss passes that train by default and are not followed by a backward pass: the next step works on the same tensors."""
    tr = _trainer()
    graph = _StepGraph(tr)
    tok, tgt = _batch(tr)
    tr.forward_backward(tok, tgt)
    graph.ran_without()
    kept, state = [weakref.ref(t) for t in graph._tensors()], graph.state
    attn = [t for t in vars(tr.engine.attn).values() if isinstance(t, (torch.Tensor, dict, list))]
    addresses = {t.data_ptr() for v in attn for t in ([v] if isinstance(v, torch.Tensor) else v.values() if isinstance(v, dict) else v)}
    assert len(addresses) == tr.cfg.n_layers + 1  # a log-sum-exp a layer, the scratch memory
    for _ in range(3):
        tr.engine.forward(tok, tgt)
        gc.collect()
        assert all(t() is not None for t in kept) and graph._state(graph._tensors()) == state
    tr.forward_backward(tok, tgt)
    assert graph._state(graph._tensors()) == state


@pytest.mark.parametrize("change", ["rope", "ws_dy", "x", "_scratch", "_lse", "norm_eps", "grad_scale", "attn"])
def test_a_change_is_seen_and_the_old_tensors_stay(change):
    tr = _trainer()
    eng, graph = tr.engine, _StepGraph(tr)
    tok, tgt = _batch(tr)
    tr.forward_backward(tok, tgt)
    graph.ran_without()
    old = weakref.ref({"rope": eng.rope, "ws_dy": eng.ws_dy, "x": eng.x[1], "_scratch": eng.attn._scratch}.get(change, eng.logits))
    if change in ("rope", "ws_dy"):
        setattr(eng, change, getattr(eng, change).clone())
    elif change == "x":
        eng.x[1] = eng.x[1].clone()
    elif change == "_scratch":
        eng.attn._scratch = eng.attn._scratch.clone()
    elif change == "_lse":
        eng.attn._lse[0] = eng.attn._lse[0].clone()
    elif change == "norm_eps":
        eng.cfg.norm_eps *= 2
    elif change == "grad_scale":
        eng.grad_scale = 0.5
    else:
        eng.attn = Tcgen05Attention(eng.cfg)
    gc.collect()
    assert old() is not None
    assert graph._state(graph._tensors()) != graph.state


class _Hooked(ShardedLlamaTrainer):
    def _grad_done(self, u):
        super()._grad_done(u)


class _Buffers(ShardedLlamaTrainer):
    def _grad_buf(self, u):
        return super()._grad_buf(u)


class _Steps(ShardedLlamaTrainer):
    def forward_backward(self, tokens, targets):  # runs around the graph, not in it
        return super().forward_backward(tokens, targets)


def _attention(cls):
    def change(tr):
        tr.engine.attn.__class__ = cls

    return change


class _Backward(Tcgen05Attention):
    def backward(self, layer, dout, batch, seq, dqkv, rope=None):
        super().backward(layer, dout, batch, seq, dqkv, rope)


@pytest.mark.parametrize("cls,change,own", [
    (ShardedLlamaTrainer, lambda tr: None, True),
    (_Steps, lambda tr: None, True),
    (_Hooked, lambda tr: None, False),
    (_Buffers, lambda tr: None, False),
    (ShardedLlamaTrainer, _attention(_Backward), False),
    (ShardedLlamaTrainer, lambda tr: setattr(tr, "manager", object()), False),
    (ShardedLlamaTrainer, lambda tr: setattr(tr, "_replica_allreduce", lambda u: None), False),
    (ShardedLlamaTrainer, lambda tr: setattr(tr.engine, "grad_done", lambda u: None), False),
    (ShardedLlamaTrainer, lambda tr: setattr(tr.engine, "_wgrad", lambda *a, **k: None), False),
    (ShardedLlamaTrainer, lambda tr: setattr(tr.engine, "forward_rows", lambda *a, **k: None), False),
    (ShardedLlamaTrainer, lambda tr: setattr(tr.engine.attn, "forward", lambda *a: None), False),
])
def test_host_code_of_others_is_not_left_out(cls, change, own):
    tr = _trainer(cls)
    graph = _StepGraph(tr)
    change(tr)
    assert graph._own_code() == own
