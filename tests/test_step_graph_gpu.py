"""The trainer's step as a CUDA graph against the same step launched kernel by kernel."""
import pytest
import torch

from torchft_b200.models.llama import CONFIGS
from torchft_b200.ops import _native as N
from torchft_b200.parallel.hsdp import ShardedLlamaTrainer

pytestmark = pytest.mark.gpu


def _batch(cfg, B, S, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    tok = torch.randint(0, cfg.vocab_size, (B, S + 1), generator=g, device="cuda")
    return tok[:, :-1], tok[:, 1:]  # not contiguous


@pytest.mark.parametrize("model,B,S,chunks", [("llama-tiny", 1, 256, 4), ("llama-small", 2, 384, 1)])
def test_graph_step_is_the_step(model, B, S, chunks):
    """New tokens, a new learning rate, loaded state, a changed gradient scale and foreign inputs on the way: losses and
    weights follow the trainer without a graph.  The two differ by the order of the atomic sums of dQ and the embedding
    gradient, which AdamW's normalisation carries into the weights: at most 2 lr an element and step, and far less in norm."""
    cfg, dev, lr = CONFIGS[model], torch.device("cuda", 0), 1e-3
    trs = [ShardedLlamaTrainer(cfg, B, S, dev, lr=lr, seed=5, logit_chunks=chunks, step_graph=on) for on in (False, True)]
    assert trs[0]._step_graph is None and trs[1]._step_graph is not None
    losses = ([], [])
    launches = []
    for step in range(8):
        kept = {k: v if k == "opt_step" else [t.clone() for t in v] for k, v in trs[0].state_dict().items()}
        for tr, out in zip(trs, losses):
            if step == 4:
                tr.lr = lr / 10
                tr.load_state_dict(kept)
            if step == 6:
                tr.engine.grad_scale = 0.5
            tok, tgt = _batch(cfg, B, S, step)
            before = N.launch_count
            out.append(tr.train_step(tok.int().long().cpu().to(dev) if step == 3 else tok, tgt))
            launches.append(N.launch_count - before)
        captured = trs[1]._step_graph.graph is not None
        assert captured == (step not in (0, 6))  # the first step, and the one after a change, run as usual
        a, b = trs[0].g_flat.float(), trs[1].g_flat.float()
        assert (a - b).norm() < 0.03 * a.norm(), step
    assert len(set(launches)) == 1  # a replay counts what it launches
    assert (torch.stack(losses[0]) - torch.stack(losses[1])).abs().max() < 0.02
    assert len({t.data_ptr() for t in losses[1]}) == 8  # every step's loss is its own tensor
    moved = 4 * lr + 4 * lr / 10
    assert (trs[0].master_flat - trs[1].master_flat).abs().max() <= 2 * moved


def test_graph_step_leaves_hooks_and_strangers_alone():
    """Host code that a step would run (a gradient hook), tokens from the CPU and a capture by the caller: no graph."""
    cfg, dev = CONFIGS["llama-tiny"], torch.device("cuda", 0)
    tr = ShardedLlamaTrainer(cfg, 1, 256, dev, seed=5)
    seen = []
    own = tr.engine.grad_done
    tr.engine.grad_done = lambda u: (seen.append(u), own(u))
    tok, tgt = _batch(cfg, 1, 256, 1)
    for _ in range(3):
        tr.forward_backward(tok, tgt)
    assert tr._step_graph.graph is None and len(seen) == 3 * cfg.n_units
    tr.engine.grad_done = own
    for _ in range(3):
        tr.forward_backward(tok, tgt)
    assert tr._step_graph.graph is not None
    want = tr.g_flat.float()
    outer = torch.cuda.CUDAGraph()
    with torch.cuda.graph(outer):
        tr.forward_backward(tok, tgt)
    tr.g_flat.zero_()
    outer.replay()
    assert (tr.g_flat.float() - want).norm() < 0.03 * want.norm()


def test_graph_step_after_passes_without_a_backward():
    """Losses measured with the engine's default argument, which trains, between the steps: the captured step's tensors are
    still its own.  Tensors of the log-sum-exps' size that are made afterwards keep their values, and gradients are those of
    launches one by one (atomic sums of dQ and the embedding gradient in another order: the bound of the step's test)."""
    cfg, dev, B, S = CONFIGS["llama-tiny"], torch.device("cuda", 0), 1, 256
    trs = [ShardedLlamaTrainer(cfg, B, S, dev, seed=5, step_graph=on) for on in (False, True)]
    for step in range(6):
        tok, tgt = _batch(cfg, B, S, step)
        for tr in trs:
            tr.train_step(tok, tgt)
        assert (trs[1]._step_graph.graph is not None) == (step not in (0, 4))
        a, b = (tr.g_flat.float() for tr in trs)
        assert (a - b).norm() < 0.03 * a.norm(), step
        for tr in trs:
            for _ in range(3):
                tr.engine.forward(tok, tgt)
        others = [torch.full((B, cfg.n_heads, S), 7.0, device=dev) for _ in range(8 * cfg.n_layers)]
        trs[1].forward_backward(tok, tgt)
        trs[0].forward_backward(tok, tgt)
        assert all(bool((t == 7.0).all()) for t in others), step
        if step == 3:
            trs[1].engine.rope = trs[1].engine.rope.clone()
            trs[1].train_step(tok, tgt)  # as usual: what it reads is elsewhere now
            assert trs[1]._step_graph.graph is None
            trs[0].train_step(tok, tgt)
            trs[1].engine.rope = trs[1].engine.rope.clone()
