"""Numerics of every sm_100a kernel against an fp32 PyTorch reference of the same op."""
import math

import pytest
import torch

from torchft_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel_err(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / (b.norm() + 1e-12)).item()


@pytest.mark.parametrize("impl", ["1cta", "2cta"])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K_", [(128, 256, 64), (256, 512, 256), (384, 768, 1024), (200, 328, 136), (1024, 1024, 4096)])
def test_gemm_layouts(a_mn, b_mn, M, N, K_, impl):
    torch.manual_seed(1)
    a = torch.randn((K_, M) if a_mn else (M, K_), device=DEV).bfloat16()
    b = torch.randn((K_, N) if b_mn else (N, K_), device=DEV).bfloat16()
    out = K.gemm(a, b, a_mn, b_mn, impl=impl)
    af = a.float().t() if a_mn else a.float()
    bf = b.float() if b_mn else b.float().t()
    ref = af @ bf
    K.check_status(out.device)
    assert rel_err(out, ref) < 1e-2
    # fp32 output + accumulate
    acc = torch.ones(M, N, device=DEV, dtype=torch.float32)
    K.gemm(a, b, a_mn, b_mn, out=acc, accumulate=True, impl=impl)
    assert rel_err(acc, ref + 1.0) < 1e-2


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("past", [-8, 0, 8, 264])
def test_gemm_tile_width(a_mn, b_mn, past):
    """On both sides of the line between 128- and 256-column tiles (the narrow ones of a row of tiles fit the CTA pairs),
    with remainders in every dimension.  Same sums in the same order either way: bf16 rounding of the result is the whole
    error (2^-9 relative)."""
    N = 128 * (torch.cuda.get_device_properties(0).multi_processor_count // 2) + past
    torch.manual_seed(9)
    M, K_ = 200, 328
    a = torch.randn((K_, M) if a_mn else (M, K_), device=DEV).bfloat16()
    b = torch.randn((K_, N) if b_mn else (N, K_), device=DEV).bfloat16()
    ref = (a.float().t() if a_mn else a.float()) @ (b.float() if b_mn else b.float().t())
    out = torch.full((M, N + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    K.gemm(a, b, a_mn, b_mn, out=out[:, :N])
    assert rel_err(out[:, :N], ref) < 4e-3 and bool((out[:, N:] == 7.0).all())
    acc = torch.ones(M, N, device=DEV, dtype=torch.float32)
    K.gemm(a, b, a_mn, b_mn, out=acc, accumulate=True)
    assert rel_err(acc, ref + 1.0) < 1e-5
    K.check_status(out.device)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K_", [
    (80, 1000, 14400),    # less than a wave of tiles; remainders in M and N
    (752, 1024, 8200),    # a share of the K slabs each, one slab short
    (1536, 4096, 9216),   # a whole wave first, then the shared tiles
    (304, 520, 5000),     # K no multiple of 8 slabs times the pairs
])
def test_gemm_split_last_wave(a_mn, b_mn, M, N, K_):
    """Tiles of the last wave that a cluster of pairs shares along K: bf16, fp32 and accumulated results, the same bits every
    time.  fp32 sums of K products in another order: sqrt(K) * 2^-24 of the result, plus bf16 rounding where it is stored so."""
    torch.manual_seed(M)
    a = torch.randn((K_, M) if a_mn else (M, K_), device=DEV).bfloat16()
    b = torch.randn((K_, N) if b_mn else (N, K_), device=DEV).bfloat16()
    ref = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    out = torch.full((M, N + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    K.gemm(a, b, a_mn, b_mn, out=out[:, :N])
    assert bool((out[:, N:] == 7.0).all()) and rel_err(out[:, :N], ref) < 2**-9
    assert torch.equal(out[:, :N], K.gemm(a, b, a_mn, b_mn))
    acc = torch.ones(M, N, device=DEV, dtype=torch.float32)
    K.gemm(a, b, a_mn, b_mn, out=acc, accumulate=True)
    assert ((acc - 1.0).double() - ref).norm() <= 4 * K_**0.5 * 2**-24 * ref.norm()
    both = out[:, :N].clone()
    K.gemm(a, b, a_mn, b_mn, out=both, accumulate=True)
    assert rel_err(both, 2 * ref) < 2**-8
    K.check_status(out.device)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (True, True)])
@pytest.mark.parametrize("M,N,K_", [(8, 8, 64), (40, 72, 200), (256, 128, 64), (264, 136, 72), (296, 520, 264), (8192, 1024, 752),
                                    (1024, 264, 3000), (752, 1024, 8200), (5000, 2056, 64)])
def test_gemm_adds_to_bf16(M, N, K_, a_mn, b_mn):
    """What C holds comes and goes by TMA, shared tiles excepted: the sum with the fp32 product, rounded once, to the bit, and
    nothing beyond M and N."""
    torch.manual_seed(M + N)
    a = torch.randn((K_, M) if a_mn else (M, K_), device=DEV).bfloat16()
    b = torch.randn((K_, N) if b_mn else (N, K_), device=DEV).bfloat16()
    product = K.gemm(a, b, a_mn, b_mn, out_dtype=torch.float32)
    out = (torch.randn(M + 3, N + 16, device=DEV) * K_**0.5).bfloat16()
    want = out.clone()
    want[:M, 8 : N + 8] = (want[:M, 8 : N + 8].float() + product).bfloat16()
    K.gemm(a, b, a_mn, b_mn, out=out[:M, 8 : N + 8], accumulate=True)
    K.check_status(out.device)
    assert torch.equal(out, want)


@pytest.mark.parametrize("N", [1, 2, 17, 1000, 8192])
@pytest.mark.parametrize("K_", [8, 72, 256, 1024, 1032, 4104])
def test_gemm_one_row(N, K_):
    """A single row reads the other operand once, by a kernel of its own; the remainders of its lanes and rows, a row stride.
    fp32 sums: bf16 rounding of the result (at most 2^-8 of each value) is the error.  Transposed operands, fp32 results and
    accumulation stay with the tiles."""
    torch.manual_seed(N + K_)
    a, b = torch.randn(1, K_, device=DEV).bfloat16(), torch.randn(N + 1, K_ + 8, device=DEV).bfloat16()[:N, :K_]
    ref = a.double() @ b.double().t()
    out = torch.full((2, N + 4), 7.0, device=DEV, dtype=torch.bfloat16)
    K.gemm(a, b, out=out[:1, :N])
    assert ((out[0, :N].double() - ref[0]).abs() <= 2**-8 * ref[0].abs() + 1e-4).all()
    assert bool((out[1] == 7.0).all()) and bool((out[0, N:] == 7.0).all())
    acc = torch.ones(1, N, device=DEV, dtype=torch.float32)
    K.gemm(a, b, out=acc, accumulate=True)
    # K products and the one summed in fp32, in any order: K 2^-24 of the sum of their magnitudes at most
    assert ((acc.double() - 1 - ref).abs() <= (K_ + 1) * 2**-24 * (1 + a.double().abs() @ b.double().abs().t())).all()
    K.check_status(a.device)


@pytest.mark.parametrize("M", [1, 33, 160, 257])
@pytest.mark.parametrize("N", [8, 72, 200, 328, 12])
def test_gemm_store_edges(M, N):
    """Outputs that end inside the epilogue's 32-row, 64-column pieces, with and without the fused activation, and one (12
    columns) that takes the general path: nothing beyond them is written, and the products are the same bits wherever they
    lie in a piece."""
    torch.manual_seed(M + N)
    a, b = torch.randn(M, 96, device=DEV).bfloat16(), torch.randn(N, 96, device=DEV).bfloat16()
    out = torch.full((M + 1, N + 12 - N % 8), 7.0, device=DEV, dtype=torch.bfloat16)
    K.gemm(a, b, out=out[:M, :N])
    assert bool((out[M:] == 7.0).all()) and bool((out[:, N:] == 7.0).all())
    # further rows and columns of tiles: other pieces, the same values
    big = K.gemm(torch.cat([a, a]), torch.cat([b, b]))
    assert torch.equal(out[:M, :N], big[M:, N:] if N % 8 == 0 else big[:M, :N])
    assert rel_err(out[:M, :N], a.float() @ b.float().t()) < 2**-8
    if N % 32 == 8:
        N2 = 32 * (N // 8)
        w = torch.randn(N2, 96, device=DEV).bfloat16()
        gu, act = (torch.full((M + 1, n + 8), 7.0, device=DEV, dtype=torch.bfloat16) for n in (N2, N2 // 2))
        K.linear_swiglu_fwd(a, w, gu[:M, :N2], act[:M, : N2 // 2])
        assert torch.equal(gu[:M, :N2], K.gemm(a, w)) and torch.equal(act[:M, : N2 // 2], K.swiglu_fwd(gu[:M, :N2].contiguous()))
        for t, n in ((gu, N2), (act, N2 // 2)):
            assert bool((t[M:] == 7.0).all()) and bool((t[:, n:] == 7.0).all())
    K.check_status(a.device)


@pytest.mark.parametrize("impl", ["1cta", "2cta"])
def test_gemm_many_tiles_persistent(impl):
    torch.manual_seed(2)
    M, N, K_ = 2048, 4096, 512
    a = torch.randn(M, K_, device=DEV).bfloat16()
    b = torch.randn(N, K_, device=DEV).bfloat16()
    ref = a.float() @ b.float().t()
    for ctas in (0, 7, 1):
        out = K.gemm(a, b, max_ctas=ctas, impl=impl)
        assert rel_err(out, ref) < 1e-2
    K.check_status(a.device)


def test_linear_trio_matches_autograd():
    torch.manual_seed(3)
    T, Kd, Nd = 512, 384, 640
    x = torch.randn(T, Kd, device=DEV).bfloat16()
    w = (torch.randn(Nd, Kd, device=DEV) * 0.05).bfloat16()
    dy = torch.randn(T, Nd, device=DEV).bfloat16()
    assert rel_err(K.linear_fwd(x, w), x.float() @ w.float().t()) < 1e-2
    assert rel_err(K.linear_dgrad(dy, w), dy.float() @ w.float()) < 1e-2
    assert rel_err(K.linear_wgrad(dy, x), dy.float().t() @ x.float()) < 1e-2


@pytest.mark.parametrize("T,D", [(64, 256), (33, 4096), (7, 1024), (701, 4096), (613, 8192)])
def test_rmsnorm(T, D):
    torch.manual_seed(4)
    x = torch.randn(T, D, device=DEV).bfloat16()
    res = torch.randn(T, D, device=DEV).bfloat16()
    w = (1 + 0.1 * torch.randn(D, device=DEV)).bfloat16()
    out, rstd, _ = K.rmsnorm_fwd(x, w, 1e-5)
    ro, rr, _ = K.ref_rmsnorm_fwd(x, w, 1e-5)
    assert rel_err(out, ro) < 1e-2 and rel_err(rstd, rr) < 1e-4
    out2, rstd2, h = K.rmsnorm_fwd(x, w, 1e-5, res=res)
    ro2, rr2, rh = K.ref_rmsnorm_fwd(x, w, 1e-5, res)
    assert rel_err(out2, ro2) < 1e-2 and rel_err(h, rh) < 1e-2
    dy = torch.randn(T, D, device=DEV).bfloat16()
    dres = torch.randn(T, D, device=DEV).bfloat16()
    dx, dw = K.rmsnorm_bwd(dy, x, w, rstd, dres=dres)
    rdx, rdw = K.ref_rmsnorm_bwd(dy, x, w, rr, dres)
    assert rel_err(dx, rdx) < 1e-2
    assert rel_err(dw, rdw) < 2e-2


@pytest.mark.parametrize("T", [1, 5, 149, 1300])
@pytest.mark.parametrize("D", [8, 256, 264, 520, 1032, 2048, 2304, 8192, 8200])
def test_rmsnorm_row_shapes(T, D):
    """Every number of warps a row, full and with a remainder, few rows and more than the groups of a pass; beyond 8192
    elements the forward pass reads its rows twice and the backward pass refuses.  The sums are fp32 (a few 2^-24 of sqrt(D)
    terms), so bf16 rounding of the results is the error: at most 2^-8 of each value."""
    torch.manual_seed(T + D)
    x, res, dy, dres = (torch.randn(T, D, device=DEV).bfloat16() for _ in range(4))
    w = (1 + 0.1 * torch.randn(D, device=DEV)).bfloat16()
    h, out = torch.empty_like(x), torch.empty_like(x)
    _, rstd, _ = K.rmsnorm_fwd(x, w, 1e-5, res=res, h_out=h, out=out)
    assert torch.equal(h, (x.float() + res.float()).bfloat16())
    ro, rr, _ = K.ref_rmsnorm_fwd(h, w, 1e-5)
    assert rel_err(out, ro.float()) < 2**-8 and rel_err(rstd, rr) < 1e-6
    assert torch.equal(K.rmsnorm_fwd(h, w, 1e-5, want_out=False)[1], rstd)
    if D > 8192:
        with pytest.raises(K.N.KernelError):
            K.rmsnorm_bwd(dy, h, w, rstd, dres=dres)
        return
    for extra in (None, dres):
        dw = torch.ones(D, device=DEV).bfloat16()
        dx, _ = K.rmsnorm_bwd(dy, h, w, rstd, dres=extra, dw=dw, accumulate_dw=True)
        hd, dyd, wd, r = h.double(), dy.double(), w.double(), rr.double().unsqueeze(-1)
        want = r * wd * dyd - hd * (dyd * wd * hd).sum(-1, keepdim=True) * r**3 / D + (0 if extra is None else extra.double())
        assert rel_err(dx, want) < 2**-8 and rel_err(dw, 1 + (dyd * hd * r).sum(0)) < 2**-8


def test_rope_roundtrip_and_ref():
    torch.manual_seed(5)
    S, Hq, Hkv, Dh = 64, 4, 2, 64
    T = 2 * S
    buf = torch.randn(T, (Hq + 2 * Hkv) * Dh, device=DEV).bfloat16()
    orig = buf.clone()
    table = K.rope_table(S, Dh, 500000.0, DEV)
    ref = K.ref_rope(orig, table, S, Hq + Hkv, Dh)
    K.rope_(buf, table, S, Hq + Hkv, Dh)
    assert rel_err(buf, ref) < 1e-2
    assert torch.equal(buf[:, (Hq + Hkv) * Dh:], orig[:, (Hq + Hkv) * Dh:])
    K.rope_(buf, table, S, Hq + Hkv, Dh, backward=True)
    assert rel_err(buf, orig) < 2e-2


def test_swiglu():
    torch.manual_seed(6)
    T, Fd = 96, 512
    gu = torch.randn(T, 2 * Fd, device=DEV).bfloat16()
    ds = torch.randn(T, Fd, device=DEV).bfloat16()
    assert rel_err(K.swiglu_fwd(gu), K.ref_swiglu_fwd(gu)) < 1e-2
    ref = K.ref_swiglu_bwd(ds, gu)
    got = K.swiglu_bwd(ds, gu.clone())
    assert rel_err(got, ref) < 1e-2
    inplace = gu.clone()
    K.swiglu_bwd(ds, inplace, dgu=inplace)
    assert rel_err(inplace, ref) < 1e-2


@pytest.mark.parametrize("T,V", [(16, 1024), (5, 128256), (64, 8192)])
def test_cross_entropy(T, V):
    torch.manual_seed(7)
    logits = (torch.randn(T, V, device=DEV) * 3).bfloat16()
    tgt = torch.randint(0, V, (T,), device=DEV)
    rl, rg = K.ref_cross_entropy(logits, tgt, 1.0 / T)
    loss = K.cross_entropy_(logits, tgt, 1.0 / T)
    assert rel_err(loss, rl) < 1e-3
    assert rel_err(logits, rg) < 1e-2


@pytest.mark.parametrize("V", [8, 4088, 4096, 4104, 4 * 4096 - 8, 4 * 4096, 4 * 4096 + 8, 7 * 4096 + 2000])
def test_cross_entropy_row_lengths(V):
    """Rows that end inside a thread's batch of loads, targets at both ends.  A gradient rounds to bf16 (8
    significant bits: half a unit of the last is up to 2^-8 of the value) after a handful of fp32 operations on numbers of at
    most 1 (2^-20 of them, the exponential's error included)."""
    T = 5
    wide = torch.randn(T, V + 16, device="cuda").mul_(4).bfloat16()
    logits = wide[:, :V]
    tgt = torch.tensor([0, V - 1, -1, V // 2, 7], device="cuda")
    x = logits.double()
    loss = K.cross_entropy_(logits, tgt, 0.5)
    onehot = torch.nn.functional.one_hot(tgt.clamp(min=0), V).double()
    want = (x.softmax(-1) - onehot) * 0.5 * (tgt >= 0)[:, None]
    assert bool(((logits.double() - want).abs() <= 2**-8 * want.abs() + 2**-20).all())
    ref = (x.logsumexp(-1) - (x * onehot).sum(-1)) * (tgt >= 0)
    assert bool(((loss.double() - ref).abs() <= 2**-18 * (1 + x.abs().amax(-1))).all())


@pytest.mark.parametrize("V", [8, 8 * 1024, 8 * 1024 + 8, 8 * 3 * 1024 - 8, 128256])
def test_cross_entropy_without_gradient(V):
    """One to several vectors per thread, with remainders; the logits stay as they are and the loss is the same number."""
    torch.manual_seed(10)
    logits = (torch.randn(3, V, device=DEV) * 3).bfloat16()
    tgt = torch.tensor([0, V - 1, -1], device=DEV)
    kept = logits.clone()
    loss = K.cross_entropy_(logits, tgt, 1.0, grad=False)
    assert torch.equal(logits, kept) and loss[2] == 0
    want = torch.nn.functional.cross_entropy(kept.double(), tgt.clamp(min=0), reduction="none")[:2]
    assert rel_err(loss[:2], want) < 1e-5  # fp32 sums of V terms
    assert torch.equal(K.cross_entropy_(logits, tgt, 1.0), loss)
    assert rel_err(logits[:2], K.ref_cross_entropy(kept, tgt.clamp(min=0), 1.0)[1][:2]) < 1e-2 and not logits[2].any()


@pytest.mark.parametrize("T,Kd,F", [(1, 2048, 8), (33, 2056, 40), (200, 2048, 512), (1000, 2048, 2816), (130, 4096, 1000), (300, 64, 128)])
def test_linear_dswiglu(T, Kd, F):
    """Down projection and activation backwards in one kernel against 64 bits: the gradient of the activation is not rounded on
    the way, so the result's rounding (at most 2^-8 of each value) is the whole error."""
    torch.manual_seed(T + F)
    dy, w = torch.randn(T, Kd, device=DEV).bfloat16(), (0.05 * torch.randn(Kd, F, device=DEV)).bfloat16()
    buf = torch.full((T + 1, 2 * F + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    gu = torch.randn(T, 2 * F, device=DEV).bfloat16()
    buf[:T, : 2 * F] = gu
    ds = torch.empty(T, F, device=DEV, dtype=torch.bfloat16)
    if Kd < 2048:  # the two kernels, which want their pairs in one piece
        with pytest.raises(ValueError):
            K.linear_dswiglu_(dy, w, buf[:T, : 2 * F], ds)
        whole = gu.clone()
        K.linear_dswiglu_(dy, w, whole, ds)
        buf[:T, : 2 * F] = whole
    else:
        K.linear_dswiglu_(dy, w, buf[:T, : 2 * F], ds)
    g, u, d = gu[:, 0::2].double(), gu[:, 1::2].double(), dy.double() @ w.double()
    sg = torch.sigmoid(g)
    want = torch.stack([d * u * (sg + g * sg * (1 - sg)), d * g * sg], dim=-1).reshape(T, 2 * F)
    assert rel_err(buf[:T, : 2 * F], want) < 2**-8
    assert bool((buf[T:] == 7.0).all()) and bool((buf[:, 2 * F :] == 7.0).all())
    K.check_status(dy.device)


@pytest.mark.parametrize("T,Kd,V", [(37, 128, 1000), (300, 256, 8192), (129, 64, 20008), (1050, 72, 1000), (131080, 64, 8)])
def test_linear_cross_entropy(T, Kd, V):
    """Head product and loss without stored logits against the two kernels: ignored targets and targets beyond the vocabulary
    count alike, a NaN in one row stays there.  Sums of V exponentials in fp32, in another order: 1e-5."""
    torch.manual_seed(V)
    x, w = torch.randn(T, Kd, device=DEV).bfloat16(), (0.2 * torch.randn(V, Kd, device=DEV)).bfloat16()
    tgt = torch.randint(0, V, (T,), device=DEV)
    tgt[T // 3] = -1
    if T > 2:
        tgt[T // 2] = V + 3
        x[T - 1, 0] = float("nan")
    plain = K.linear_fwd(x, w)
    want = K.cross_entropy_(plain.clone(), tgt, 0.25, grad=False)
    loss = torch.empty(T, device=DEV)
    K.linear_cross_entropy_(x, w, tgt, 0.25, torch.empty_like(plain), loss, grad=False)
    K.check_status(x.device)
    torch.testing.assert_close(loss, want, rtol=1e-5, atol=1e-5, equal_nan=True)
    both = torch.empty_like(plain)
    K.linear_cross_entropy_(x, w, tgt, 0.25, both, loss, grad=True)
    torch.testing.assert_close(loss, want, rtol=1e-5, atol=1e-5, equal_nan=True)
    assert torch.equal(K.cross_entropy_(plain, tgt, 0.25).isfinite(), loss.isfinite())
    assert torch.equal(plain.nan_to_num(), both.nan_to_num())


@pytest.mark.parametrize("gdt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [8, 1000, 1 << 20, (1 << 20) + 3])
def test_adamw(gdt, n):
    torch.manual_seed(8)
    master = torch.randn(n, device=DEV)
    m = torch.zeros(n, device=DEV)
    v = torch.zeros(n, device=DEV)
    lp = torch.empty(n, device=DEV, dtype=torch.bfloat16)
    rm, rmm, rv = master.clone(), m.clone(), v.clone()
    scale = torch.tensor([0.5], device=DEV)
    for step in (1, 2, 3):
        g = torch.randn(n, device=DEV).to(gdt)
        K.adamw_(master, m, v, g, lp, 1e-2, 0.9, 0.95, 1e-8, 0.1, step, scale)
        K.ref_adamw(rm, rmm, rv, g, 1e-2, 0.9, 0.95, 1e-8, 0.1, step, 0.5)
    assert rel_err(master, rm) < 1e-5
    assert rel_err(m, rmm) < 1e-5 and rel_err(v, rv) < 1e-5
    assert torch.equal(lp, master.bfloat16())


def test_sumsq_and_clip():
    torch.manual_seed(9)
    x = torch.randn((1 << 18) + 5, device=DEV).bfloat16()
    out = torch.zeros(1, device=DEV)
    K.sumsq_(x, out)
    ref = x.float().pow(2).sum()
    assert abs(out.item() - ref.item()) / ref.item() < 1e-4
    coef = torch.zeros(1, device=DEV)
    nrm = torch.zeros(1, device=DEV)
    K.clip_coef_(out, 1.0, coef, nrm)
    assert abs(nrm.item() - math.sqrt(ref.item())) / nrm.item() < 1e-4
    assert abs(coef.item() - 1.0 / (nrm.item() + 1e-6)) < 1e-6


def test_embedding():
    torch.manual_seed(10)
    V, D, T = 512, 256, 300
    table = torch.randn(V, D, device=DEV).bfloat16()
    tok = torch.randint(0, V, (T,), device=DEV)
    assert torch.equal(K.embedding_fwd(tok, table), table[tok])
    dout = torch.randn(T, D, device=DEV).bfloat16()
    dtab = torch.zeros(V, D, device=DEV, dtype=torch.bfloat16)
    K.embedding_bwd(tok, dout, dtab)
    ref = torch.zeros(V, D, device=DEV).index_add_(0, tok, dout.float())
    assert rel_err(dtab, ref) < 2e-2


@pytest.mark.parametrize("variant", ["library", "head_dim_128", "head_dim_64"])
def test_engine_matches_autograd_gpu(variant):
    from torchft_b200.models.llama import LLAMA_TINY, LlamaConfig, SdpaAttention, Tcgen05Attention, TorchLlama, _Fields
    from torchft_b200.parallel.hsdp import ShardedLlamaTrainer

    torch.manual_seed(0)
    # the tcgen05 attention kernels take head dim 128, and head dim 64 (LLAMA_TINY) when the sequence is a multiple
    # of 256; LLAMA_TINY at sequence 128 falls back to the library
    cfg = (LlamaConfig(dim=256, n_layers=2, n_heads=2, n_kv_heads=1, ffn_dim=512, vocab_size=1024, name="llama-hd128")
           if variant == "head_dim_128" else LLAMA_TINY)
    B, S = 2, (256 if variant == "head_dim_64" else 128)
    native_attention = variant != "library"
    dev = torch.device("cuda")
    tr = ShardedLlamaTrainer(cfg, B, S, dev, logit_chunks=2)
    assert isinstance(tr.engine.attn, Tcgen05Attention if native_attention else SdpaAttention)
    tokens = torch.randint(0, cfg.vocab_size, (B, S), device=dev)
    targets = torch.randint(0, cfg.vocab_size, (B, S), device=dev)
    loss = tr.forward_backward(tokens, targets)
    ref = TorchLlama(cfg).to(dev, torch.float32)
    ref.load_units(lambda u: tr._param_unit(u))
    rl = torch.nn.functional.cross_entropy(ref(tokens).float().view(-1, cfg.vocab_size), targets.view(-1))
    rl.backward()
    K.check_status(dev)
    assert abs(loss.item() - rl.item()) < 3e-2
    g = _Fields(tr._grad_unit(1), cfg.unit_fields(1))
    for name in ("wqkv", "wo", "wgu", "wd", "attn_norm", "ffn_norm"):
        assert rel_err(getattr(g, name), getattr(ref.layers[0], name).grad) < 0.03, name
    l0 = loss.item()
    for _ in range(3):
        tr.optimizer_step()
        l1 = tr.forward_backward(tokens, targets).item()
    assert l1 < l0


def test_engine_matches_autograd_at_the_8b_layer_shape():
    """One decoder layer with the shapes the benchmark runs (dim 4096, ffn 14336, 32 query heads on 8 KV heads,
    sequence 8192: reductions of depth 4096, 8192 and 14336, attention over 64 key blocks) against fp32 autograd.
    The vocabulary is cut to 8192 to bound the oracle's memory."""
    from torchft_b200.models.llama import LlamaConfig, Tcgen05Attention, TorchLlama, _Fields
    from torchft_b200.parallel.hsdp import ShardedLlamaTrainer

    torch.manual_seed(0)
    torch.backends.cuda.matmul.allow_tf32 = False
    cfg = LlamaConfig(dim=4096, n_layers=1, n_heads=32, n_kv_heads=8, ffn_dim=14336, vocab_size=8192, name="llama-8b-layer")
    B, S = 1, 8192
    dev = torch.device("cuda")
    tr = ShardedLlamaTrainer(cfg, B, S, dev, logit_chunks=1)
    assert isinstance(tr.engine.attn, Tcgen05Attention)
    tokens = torch.randint(0, cfg.vocab_size, (B, S), device=dev)
    targets = torch.randint(0, cfg.vocab_size, (B, S), device=dev)
    loss = tr.forward_backward(tokens, targets)
    K.check_status(dev)
    ref = TorchLlama(cfg).to(dev, torch.float32)
    ref.load_units(lambda u: tr._param_unit(u))
    rl = torch.nn.functional.cross_entropy(ref(tokens).float().view(-1, cfg.vocab_size), targets.view(-1))
    rl.backward()
    assert abs(loss.item() - rl.item()) < 2e-2, (loss.item(), rl.item())
    g = _Fields(tr._grad_unit(1), cfg.unit_fields(1))
    errs = {name: rel_err(getattr(g, name), getattr(ref.layers[0], name).grad)
            for name in ("wqkv", "wo", "wgu", "wd", "attn_norm", "ffn_norm")}
    print("gradient errors at the 8B layer shape:", {k: round(v, 5) for k, v in errs.items()})
    for name, e in errs.items():
        assert e < 0.02, (name, errs)


@pytest.mark.parametrize("T,Fd", [(384, 352), (1000, 1616)])  # narrow tiles; wide ones (4 x 26 narrow ones would not fit a wave)
def test_linear_swiglu_fused_epilogue(T, Fd):
    torch.manual_seed(11)
    Kd = 256  # 2F is 22 * 32 or 101 * 32
    x = torch.randn(T, Kd, device=DEV).bfloat16()
    w = (torch.randn(2 * Fd, Kd, device=DEV) * 0.1).bfloat16()
    gu = torch.empty(T, 2 * Fd, device=DEV, dtype=torch.bfloat16)
    s = torch.empty(T, Fd, device=DEV, dtype=torch.bfloat16)
    K.linear_swiglu_fwd(x, w, gu, s)
    K.check_status(x.device)
    ref_gu = x.float() @ w.float().t()
    assert rel_err(gu, ref_gu) < 1e-2
    assert rel_err(s, K.ref_swiglu_fwd(gu)) < 1e-2
    assert rel_err(s, torch.nn.functional.silu(ref_gu[:, 0::2]) * ref_gu[:, 1::2]) < 2e-2


@pytest.mark.parametrize("M,N", [(256, 512), (1000, 3232)])  # narrow tiles; wide ones
@pytest.mark.parametrize("world", [1, 3])
def test_gemm_scatter_epilogue(world, M, N):
    """The result as one field of a flat unit that `world` ranks share: every piece lands in its owner's staging area (here
    all on this GPU: the kernel only sees pointers), in the slice of the rank that computed it, and nothing else changes."""
    import ctypes

    torch.manual_seed(8)
    K_, src, unit_off = 328, world - 1, 8 * 77
    shard = -(-(unit_off + M * N + 8 * 5) // (world * 8)) * 8
    a = torch.randn(K_, M, device=DEV).bfloat16()  # both operands as a weight gradient has them
    b = torch.randn(K_, N, device=DEV).bfloat16()
    stages = [torch.full((world, shard), 7.0, device=DEV, dtype=torch.bfloat16) for _ in range(world)]
    peers = (ctypes.c_void_p * 8)()
    for r in range(world):
        peers[r] = stages[r].data_ptr()
    K.gemm_scatter(a, b, True, True, K.ScatterField(peers, world, src, shard, unit_off, (M, N)))
    K.check_status(a.device)
    unit = torch.cat([s[src] for s in stages])
    assert torch.equal(unit[unit_off : unit_off + M * N].view(M, N), K.gemm(a, b, True, True))
    assert rel_err(unit[unit_off : unit_off + M * N].view(M, N), a.float().t() @ b.float()) < 4e-3
    assert torch.all(unit[:unit_off] == 7.0) and torch.all(unit[unit_off + M * N :] == 7.0)
    assert all(torch.all(s[r] == 7.0) for s in stages for r in range(world) if r != src)


@pytest.mark.parametrize("world", [2, 4])
@pytest.mark.parametrize("M,N,K_,swiglu", [(256, 256, 64, False), (1024, 1536, 512, False), (2048, 2048, 1024, True),
                                           (200, 640, 192, False)])
def test_gemm_with_fused_all_gather(world, M, N, K_, swiglu):
    """The weight lies spread over `world` shard buffers (here all on this GPU: the kernel only sees pointers) at an
    offset that makes it straddle shard boundaries; the GEMM gathers it into the local unit while it multiplies."""
    import ctypes

    torch.manual_seed(7)
    unit_off = 8 * 331  # some field in front of the weight
    numel = unit_off + N * K_ + 8 * 57
    shard = -(-numel // (world * 8)) * 8
    shard = max(shard, 8192)
    unit = torch.zeros(shard * world, device=DEV, dtype=torch.bfloat16)
    unit[:numel] = (torch.randn(numel, device=DEV) * 0.5).bfloat16()
    shards = [unit[r * shard:(r + 1) * shard].clone() for r in range(world)]
    peers = (ctypes.c_void_p * 8)()
    for r in range(world):
        peers[r] = shards[r].data_ptr()
    full = torch.full((shard * world,), 7.0, device=DEV, dtype=torch.bfloat16)  # stale content must be overwritten
    w_true = unit[unit_off:unit_off + N * K_].view(N, K_)
    sync = torch.full((1 + N // 128,), 12345, device=DEV, dtype=torch.int32)  # the launcher zeroes it
    field = K.GatherField(full[unit_off:unit_off + N * K_].view(N, K_), peers, world, shard, unit_off, sync)
    assert K.GatherField.supported((N, K_), shard)
    x = torch.randn(M, K_, device=DEV).bfloat16()
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    if swiglu:
        s_out = torch.empty(M, N // 2, device=DEV, dtype=torch.bfloat16)
        K.linear_swiglu_fwd(x, field, out, s_out)
    else:
        K.linear_fwd(x, field, out=out)
    torch.cuda.synchronize()
    K.check_status(out.device)
    assert not field.pending
    assert torch.equal(field.local, w_true)
    assert torch.all(full[:unit_off] == 7.0) and torch.all(full[unit_off + N * K_:] == 7.0)  # nothing outside the field
    ref = x.float() @ w_true.float().t()
    assert rel_err(out, ref) < 1e-2
    if swiglu:
        g, u = out.float()[:, 0::2], out.float()[:, 1::2]
        assert rel_err(s_out, torch.nn.functional.silu(g) * u) < 1e-2
    # second use: an ordinary GEMM on the gathered weight
    out2 = K.linear_fwd(x, field)
    assert torch.equal(out2, out)
