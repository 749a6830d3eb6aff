"""Kernels may become resident while the one before them on the stream drains; what they read and write must not show it."""

import pytest
import torch

from torchft_b200.ops import kernels as K

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


class _Chain:
    """Forward and backward kernels in turn, each reading what the one before wrote, many writing what earlier ones read.
    Sequences of one key block: every sum has one order."""

    def __init__(self, batch, seq, dim, ffn, head=64, seed=0):
        g = torch.Generator(device="cuda").manual_seed(seed)
        T, D, F = batch * seq, dim, ffn
        r = lambda *shape: (torch.randn(*shape, device="cuda", generator=g) * 0.1).bfloat16()  # noqa: E731
        e = lambda *shape: torch.zeros(*shape, device="cuda", dtype=torch.bfloat16)  # noqa: E731
        self.sizes = batch, seq, dim, head
        self.x, self.h, self.w, self.wq, self.wo, self.wu, self.wd = (r(T, D), r(T, D), r(D) + 1, r(3 * D, D), r(D, D), r(2 * F, D),
                                                                      r(D, F))
        self.n, self.qkv, self.dqkv, self.gu, self.act, self.d, self.out = (e(T, D), e(T, 3 * D), e(T, 3 * D), e(T, 2 * F), e(T, F),
                                                                            e(T, D), e(T, D))
        self.dwq, self.dw = e(3 * D, D), e(D)
        self.rstd, self.lse = torch.zeros(T, device="cuda"), torch.zeros(batch, D // head, seq, device="cuda")
        self.table = K.rope_table(seq, head, 10000.0, "cuda")
        torch.cuda.synchronize()

    def step(self, between=lambda: None, side=None):
        B, S, D, hd = self.sizes
        H = D // hd
        views = lambda t: (t[:, :D], t[:, D : 2 * D], t[:, 2 * D :])  # noqa: E731
        main = torch.cuda.current_stream()
        side = side or main
        for launch in (
            lambda: K.rmsnorm_fwd(self.x, self.w, res=self.h, h_out=self.h, out=self.n, rstd=self.rstd),
            lambda: K.linear_fwd(self.n, self.wq, self.qkv),
            lambda: K.rope_(self.qkv, self.table, S, 2 * H, hd),
            lambda: K.attention_fwd(*views(self.qkv), B, S, H, H, hd, self.out, self.lse, any_length=True),
            lambda: K.linear_fwd(self.out, self.wo, self.d),
            lambda: K.linear_fwd(self.d, self.wu, self.gu),
            lambda: K.swiglu_fwd(self.gu, self.act),
            lambda: K.linear_fwd(self.act, self.wd, self.d),
            lambda: K.attention_bwd(*views(self.qkv), self.out, self.d, self.lse, *views(self.dqkv), B, S, H, H, hd, rope=self.table,
                                    any_length=True),
        ):
            launch()
            between()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            K.linear_wgrad(self.dqkv, self.n, self.dwq)
        between()
        K.linear_dgrad(self.dqkv, self.wq, self.d)
        between()
        K.rmsnorm_bwd(self.d, self.h, self.w, self.rstd, dres=self.d, dx=self.x, dw=self.dw)
        between()
        main.wait_stream(side)
        self.wq.add_(self.dwq, alpha=1e-3).clamp_(-0.3, 0.3)  # library kernels in the row; nothing grows from step to step
        self.x.clamp_(-1, 1)
        self.h.clamp_(-1, 1)

    def state(self):
        return {k: v for k, v in vars(self).items() if isinstance(v, torch.Tensor)}


@pytest.mark.parametrize("how", ["stream", "two streams", "graph"])
@pytest.mark.parametrize("sizes", [(1, 32, 64, 128), (5, 100, 256, 512), (16, 128, 512, 1536), (9, 128, 512, 1024, 128)])
def test_results_are_those_of_launches_one_by_one(sizes, how):
    STEPS = 8
    apart, run = _Chain(*sizes), _Chain(*sizes)
    for _ in range(STEPS):
        apart.step(torch.cuda.synchronize)
    side = None if how == "stream" else torch.cuda.Stream()
    if how == "graph":
        spare = _Chain(*sizes)
        spare.step(side=side)  # loads the kernels, allocates their scratch
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run.step(side=side)
        for _ in range(STEPS):
            graph.replay()
    else:
        for _ in range(STEPS):
            run.step(side=side)
    torch.cuda.synchronize()
    K.check_status(run.x.device)
    got = run.state()
    for name, want in apart.state().items():
        assert bool(want.isfinite().all()), name
        assert torch.equal(want, got[name]), name


def test_norm_gradients_on_two_streams():
    """Backward passes of norms of one width on two streams at once give what they give one after the other: no sum has
    another order, so to the bit."""
    T, D, N = 2048, 1024, 40
    g = torch.Generator(device="cuda").manual_seed(3)
    sides = []
    for _ in range(2):
        dy, x = (torch.randn(T, D, device="cuda", generator=g).bfloat16() for _ in range(2))
        sides.append((dy, x, torch.ones(D, device="cuda").bfloat16(), torch.rand(T, device="cuda", generator=g) + 0.5))
    want = [K.rmsnorm_bwd(*s) for s in sides]
    out = [[(torch.empty_like(s[1]), torch.empty_like(s[2])) for _ in range(N)] for s in sides]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in sides]
    for i in range(N):
        for s, st, o in zip(sides, streams, out):
            with torch.cuda.stream(st):
                K.rmsnorm_bwd(*s, dx=o[i][0], dw=o[i][1])
    torch.cuda.synchronize()
    for (dx, dw), o in zip(want, out):
        for got_dx, got_dw in o:
            assert torch.equal(got_dx, dx) and torch.equal(got_dw, dw)


class _Engine:
    """The engine's order around a workspace that two streams use: a kernel of one stream writes it and the other's next kernel, a
    dependent of the one before it there, waits for nothing but an event; then the first stream's next dependent overwrites what
    the other reads, again behind an event alone."""

    B, S, D, HD = 64, 128, 1024, 64

    def __init__(self, steps):
        g = torch.Generator(device="cuda").manual_seed(1)
        T, D = self.B * self.S, self.D
        r = lambda *shape: (torch.randn(*shape, device="cuda", generator=g) * 0.1).bfloat16()  # noqa: E731
        self.w, self.wo, self.wq, self.qkv, self.dqkv, self.d = r(D) + 1, r(D, D), r(3 * D, D), r(T, 3 * D), r(T, 3 * D), r(T, D)
        self.n, self.out, self.dout = (torch.zeros_like(self.d) for _ in range(3))
        self.lse = torch.zeros(self.B, D // self.HD, self.S, device="cuda")
        self.dw = [torch.zeros(3 * D, D, device="cuda", dtype=torch.bfloat16) for _ in range(steps)]
        views, H = self.views(self.qkv), D // self.HD
        K.attention_fwd(*views, self.B, self.S, H, H, self.HD, self.out, self.lse, any_length=True)
        torch.cuda.synchronize()

    def views(self, t):
        return t[:, : self.D], t[:, self.D : 2 * self.D], t[:, 2 * self.D :]

    def run(self, side=None, product=True, between=lambda: None):
        main, H = torch.cuda.current_stream(), self.D // self.HD
        side = side or main
        for dw in self.dw:
            K.rmsnorm_fwd(self.d, self.w, out=self.n)
            between()
            ready = main.record_event()
            with torch.cuda.stream(side):
                side.wait_event(ready)
                K.linear_wgrad(self.dqkv, self.n, out=dw)
                between()
                done = side.record_event()
            if product:
                K.linear_fwd(self.n, self.wo, out=self.dout)
                between()
            main.wait_event(done)
            K.attention_bwd(*self.views(self.qkv), self.out, self.dout if product else self.d, self.lse, *self.views(self.dqkv), self.B,
                            self.S, H, H, self.HD, any_length=True)
            between()
            K.linear_dgrad(self.dqkv, self.wq, out=self.d)
            between()


@pytest.mark.parametrize("product", [True, False])
@pytest.mark.parametrize("graph", [False, True])
def test_dependents_behind_an_event_alone(graph, product):
    """Sequences of one key block: every sum has one order, so the results are those of launches one by one, to the bit."""
    apart, run, side = _Engine(6), _Engine(6), torch.cuda.Stream()
    apart.run(None, product, torch.cuda.synchronize)
    if graph:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            run.run(side, product)
        g.replay()
    else:
        run.run(side, product)
    torch.cuda.synchronize()
    K.check_status(run.d.device)
    for i, (want, got) in enumerate(zip(apart.dw, run.dw)):
        assert bool(want.isfinite().all()) and bool(want.any()) and torch.equal(want, got), i
    assert torch.equal(apart.dqkv, run.dqkv) and torch.equal(apart.d, run.d)
