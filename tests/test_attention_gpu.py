"""Numerics of the tcgen05 attention kernels against an fp32 PyTorch restatement."""
import pytest
import torch

from torchft_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


def _qkv(B, S, Hq, Hkv, D, seed=0, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    qkv = (torch.randn(B * S, (Hq + 2 * Hkv) * D, device="cuda", generator=g) * scale).to(torch.bfloat16)
    q = qkv[:, : Hq * D]
    k = qkv[:, Hq * D : (Hq + Hkv) * D]
    v = qkv[:, (Hq + Hkv) * D :]
    return qkv, q, k, v


@pytest.mark.parametrize("B,S,Hq,Hkv,causal,scale", [
    (1, 128, 1, 1, True, 1.0),
    (1, 256, 2, 1, True, 1.0),
    (2, 512, 4, 2, True, 1.0),
    (1, 1024, 8, 2, True, 3.0),   # large scores: the running maximum moves and O is rescaled
    (1, 384, 2, 2, False, 1.0),
])
def test_attention_fwd_matches_reference(B, S, Hq, Hkv, causal, scale):
    D = 128
    _, q, k, v = _qkv(B, S, Hq, Hkv, D, seed=S, scale=scale)
    out = torch.empty(B * S, Hq * D, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device="cuda")
    K.attention_fwd(q, k, v, B, S, Hq, Hkv, D, out, lse, causal=causal)
    K.check_status(out.device)
    q4, k4, v4 = (t.reshape(B, S, -1, D) for t in (q, k, v))
    ref = K.ref_attention(q4.float(), k4.float(), v4.float(), causal).reshape(B * S, Hq * D)
    ref_lse = K.ref_attention_lse(q4, k4, v4, causal)
    err = (out.float() - ref).norm() / ref.norm()
    assert err < 1e-2, err
    assert (out.float() - ref).abs().max() < 0.05 * max(1.0, ref.abs().max().item())
    torch.testing.assert_close(lse, ref_lse, rtol=1e-3, atol=2e-3)


@pytest.mark.parametrize("S,more_heads,two_tiles", [
    (512, 0, False),   # the last size that one wave of 128-query CTAs takes
    (512, 1, True),    # one head more
    (640, 0, False),   # beyond a wave, but no whole number of tile pairs
    (768, 0, True),
])
def test_attention_fwd_dispatch_line(monkeypatch, S, more_heads, two_tiles):
    """The forward kernel that is chosen on both sides of one wave of CTAs, whatever the number of SMs."""
    H = torch.cuda.get_device_properties(0).multi_processor_count // 4 + more_heads
    monkeypatch.delenv("FTB200_ATTN_FWD", raising=False)
    lib, called = K.N.lib(), []

    class Recorder:
        def __getattr__(self, name):
            called.append(name)
            return getattr(lib, name)

    monkeypatch.setattr(K.N, "lib", Recorder)
    _check_fwd(1, S, H, H, 128, True, 1.0, seed=S + H)
    assert called == ["ftb200_attention_fwd2" if two_tiles else "ftb200_attention_fwd"]


def _check_fwd(B, S, Hq, Hkv, D, causal, scale, seed):
    _, q, k, v = _qkv(B, S, Hq, Hkv, D, seed=seed, scale=scale)
    out = torch.empty(B * S, Hq * D, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device="cuda")
    K.attention_fwd(q, k, v, B, S, Hq, Hkv, D, out, lse, causal=causal)
    K.check_status(out.device)
    q4, k4, v4 = (t.reshape(B, S, -1, D) for t in (q, k, v))
    ref = K.ref_attention(q4.float(), k4.float(), v4.float(), causal).reshape(B * S, Hq * D)
    ref_lse = K.ref_attention_lse(q4, k4, v4, causal)
    err = (out.float() - ref).norm() / ref.norm()
    assert err < 1e-2, err
    assert (out.float() - ref).abs().max() < 0.05 * max(1.0, ref.abs().max().item())
    torch.testing.assert_close(lse, ref_lse, rtol=1e-3, atol=2e-3)


@pytest.mark.parametrize("poly", ["0", "2", "4"])
@pytest.mark.parametrize("B,S,Hq,Hkv,D,causal,scale", [
    (1, 256, 1, 1, 128, True, 1.0),
    (2, 512, 4, 2, 128, True, 1.0),
    (1, 1024, 8, 2, 128, True, 3.0),    # the running maximum moves and O is rescaled
    (1, 512, 2, 2, 128, False, 1.0),
    (1, 256, 2, 1, 64, True, 1.0),      # head dim 64 (Llama-3.2-1B)
    (2, 1024, 8, 2, 64, True, 3.0),
    (1, 768, 4, 4, 64, False, 1.0),
])
def test_attention_fwd_pair_kernel(monkeypatch, poly, B, S, Hq, Hkv, D, causal, scale):
    """The two-tiles-per-CTA forward kernel, with none, a quarter and half of the exponentials on the FMA pipe."""
    monkeypatch.setenv("FTB200_ATTN_FWD", "pair")
    monkeypatch.setenv("FTB200_ATTN_POLY", poly)
    _check_fwd(B, S, Hq, Hkv, D, causal, scale, seed=S + D)


def test_attention_fwd_at_the_benchmark_shape():
    """Sequence 8192, 32 query heads on 8 KV heads, head dim 128: the shape of the Llama-3 8B step.  The fp32
    reference is evaluated on a slice of heads to bound its memory."""
    B, S, Hq, Hkv, D = 1, 8192, 32, 8, 128
    _, q, k, v = _qkv(B, S, Hq, Hkv, D, seed=5)
    out = torch.empty(B * S, Hq * D, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device="cuda")
    K.attention_fwd(q, k, v, B, S, Hq, Hkv, D, out, lse, causal=True)
    K.check_status(out.device)
    for kvh in (0, 7):
        qs = q.reshape(B, S, Hq, D)[:, :, kvh * 4 : kvh * 4 + 2]
        ks = k.reshape(B, S, Hkv, D)[:, :, kvh : kvh + 1]
        vs = v.reshape(B, S, Hkv, D)[:, :, kvh : kvh + 1]
        ref = K.ref_attention(qs.float(), ks.float(), vs.float(), True)
        got = out.reshape(B, S, Hq, D)[:, :, kvh * 4 : kvh * 4 + 2].float()
        err = (got - ref).norm() / ref.norm()
        assert err < 1e-2, err
        ref_lse = K.ref_attention_lse(qs, ks, vs, True)
        torch.testing.assert_close(lse[:, kvh * 4 : kvh * 4 + 2], ref_lse, rtol=1e-3, atol=2e-3)


@pytest.mark.parametrize("B,S,Hq,Hkv,causal,D", [
    (1, 128, 1, 1, True, 128),
    (1, 256, 2, 1, True, 128),
    (2, 512, 4, 2, True, 128),
    (1, 384, 2, 2, False, 128),
    (1, 256, 1, 1, True, 64),       # head dim 64 (Llama-3.2-1B): the forward needs seq % 256 == 0
    (2, 512, 8, 2, True, 64),
    (1, 2048, 8, 2, True, 64),
    (1, 768, 4, 4, False, 64),
])
def test_attention_bwd_matches_reference(B, S, Hq, Hkv, causal, D):
    qkv, q, k, v = _qkv(B, S, Hq, Hkv, D, seed=7 + S)
    out = torch.empty(B * S, Hq * D, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device="cuda")
    K.attention_fwd(q, k, v, B, S, Hq, Hkv, D, out, lse, causal=causal)
    g = torch.Generator(device="cuda").manual_seed(99)
    d_o = torch.randn(B * S, Hq * D, device="cuda", generator=g).to(torch.bfloat16)
    dqkv = torch.full_like(qkv, float("nan"))
    dq, dk, dv = dqkv[:, : Hq * D], dqkv[:, Hq * D : (Hq + Hkv) * D], dqkv[:, (Hq + Hkv) * D :]
    K.attention_bwd(q, k, v, out, d_o, lse, dq, dk, dv, B, S, Hq, Hkv, D, causal=causal)
    K.check_status(out.device)
    q4, k4, v4, do4 = (t.reshape(B, S, -1, D) for t in (q, k, v, d_o))
    rq, rk, rv = K.ref_attention_bwd(q4, k4, v4, do4, causal)
    for name, got, want in (("dq", dq, rq), ("dk", dk, rk), ("dv", dv, rv)):
        want = want.reshape(B * S, -1)
        err = (got.float() - want).norm() / want.norm()
        assert err < 2e-2, (name, err)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,S,Hq,Hkv,causal,scale", [
    (1, 256, 1, 1, True, 1.0),      # blocks of two tiles and of one
    (2, 256, 3, 1, False, 1.0),     # six tiles a block, through the stages of Q and dO
    (1, 768, 8, 1, True, 3.0),      # eight heads on one; most weights are near 0 or 1
    (1, 512, 3, 3, False, 1.0),
    (3, 1280, 2, 2, True, 1.0),     # an odd number of tiles in every other block
])
def test_attention_bwd_tiles(B, S, Hq, Hkv, causal, scale, D):
    """Tiles of 128 queries at the edges of the walk over them.  Three roundings to bf16 lie on the way of every
    gradient (probabilities or dS, the forward's O behind delta, the result), each at most 2^-8 of a value and less
    than 2^-9 in norm."""
    qkv, q, k, v = _qkv(B, S, Hq, Hkv, D, seed=S + D, scale=scale)
    out = torch.empty(B * S, Hq * D, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device="cuda")
    K.attention_fwd(q, k, v, B, S, Hq, Hkv, D, out, lse, causal=causal)
    d_o = torch.randn(B * S, Hq * D, device="cuda", generator=torch.Generator(device="cuda").manual_seed(S)).to(torch.bfloat16)
    dqkv = torch.full_like(qkv, float("nan"))
    dq, dk, dv = dqkv[:, : Hq * D], dqkv[:, Hq * D : (Hq + Hkv) * D], dqkv[:, (Hq + Hkv) * D :]
    for _ in range(2):  # the second call finds the first one's sums in the scratch memory
        K.attention_bwd(q, k, v, out, d_o, lse, dq, dk, dv, B, S, Hq, Hkv, D, causal=causal)
    K.check_status(out.device)
    want = K.ref_attention_bwd(*(t.reshape(B, S, -1, D) for t in (q, k, v, d_o)), causal)
    for name, got, w in zip(("dq", "dk", "dv"), (dq, dk, dv), want):
        w = w.reshape(B * S, -1)
        assert (got.float() - w).norm() <= 3 * 2**-9 * w.norm(), name


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,Hq,Hkv", [(2, 1, 2, 1), (3, 7, 1, 1), (2, 127, 2, 2), (2, 128, 2, 1), (2, 129, 4, 2), (1, 255, 2, 1),
                                        (3, 257, 2, 2), (2, 384, 2, 1), (2, 385, 2, 1), (3, 1000, 8, 2)])
def test_attention_of_any_length(B, S, Hq, Hkv, causal, D):
    """Sequences that end inside a tile, next to each other in memory: what lies behind an end (the next sequence, NaN behind
    the last one) neither enters nor is written over.  Tolerances as for whole tiles."""
    n = (Hq + 2 * Hkv) * D
    whole = torch.full((B * S + 300, n), float("nan"), device="cuda", dtype=torch.bfloat16)
    whole[: B * S] = _qkv(B, S, Hq, Hkv, D, seed=S)[0]
    qkv = whole[: B * S]
    q, k, v = qkv[:, : Hq * D], qkv[:, Hq * D : (Hq + Hkv) * D], qkv[:, (Hq + Hkv) * D :]
    out = torch.full((B * S + 300, Hq * D), 7.0, dtype=torch.bfloat16, device="cuda")
    lse = torch.full((B * Hq * S + 300,), 7.0, device="cuda")
    with pytest.raises(K.N.KernelError) if S % 256 and (S % 128 or D == 64) else __import__("contextlib").nullcontext():
        K.attention_fwd(q, k, v, B, S, Hq, Hkv, D, out[: B * S].clone(), None, causal=causal)  # refused unless asked for
    K.attention_fwd(q, k, v, B, S, Hq, Hkv, D, out[: B * S], lse[: B * Hq * S].view(B, Hq, S), causal=causal, any_length=True)
    d_o = torch.full_like(out, float("nan"))
    d_o[: B * S] = torch.randn(B * S, Hq * D, device="cuda")
    d = torch.full_like(whole, 7.0)
    K.attention_bwd(q, k, v, out[: B * S], d_o[: B * S], lse[: B * Hq * S].view(B, Hq, S), d[: B * S, : Hq * D],
                    d[: B * S, Hq * D : (Hq + Hkv) * D], d[: B * S, (Hq + Hkv) * D :], B, S, Hq, Hkv, D, causal=causal, any_length=True)
    K.check_status(out.device)
    for t, rows in ((out, B * S), (d, B * S), (lse, B * Hq * S)):
        assert bool((t[rows:] == 7.0).all())
    q4, k4, v4, do4 = (t.reshape(B, S, -1, D) for t in (q, k, v, d_o[: B * S]))
    ref = K.ref_attention(q4.float(), k4.float(), v4.float(), causal).reshape(B * S, Hq * D)
    assert (out[: B * S].float() - ref).norm() < 1e-2 * ref.norm()
    torch.testing.assert_close(lse[: B * Hq * S].view(B, Hq, S), K.ref_attention_lse(q4, k4, v4, causal), rtol=1e-3, atol=2e-3)
    want = torch.cat([w.reshape(B * S, -1) for w in K.ref_attention_bwd(q4, k4, v4, do4, causal)], dim=1)
    if S > 1:  # a single key has no gradient but its value's
        for a, b in ((0, Hq), (Hq, Hq + Hkv), (Hq + Hkv, Hq + 2 * Hkv)):
            got, w = d[: B * S, a * D : b * D].float(), want[:, a * D : b * D]
            assert (got - w).norm() < 2e-2 * w.norm()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_attention_bwd_rotates_back(D, causal):
    """dQ and dK of the values before the rotation: as the rotated ones turned back by a kernel of their own, which rounds once
    more (at most 2^-8 of each value)."""
    B, S, Hq, Hkv = 2, 512, 4, 2
    qkv, q, k, v = _qkv(B, S, Hq, Hkv, D, seed=D)
    table = K.rope_table(S, D, 10000.0, "cuda")
    out = torch.empty(B * S, Hq * D, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device="cuda")
    K.attention_fwd(q, k, v, B, S, Hq, Hkv, D, out, lse, causal=causal)
    d_o = torch.randn_like(out)
    grads = []
    for rope in (None, table):
        d = torch.full_like(qkv, float("nan"))
        K.attention_bwd(q, k, v, out, d_o, lse, d[:, : Hq * D], d[:, Hq * D : (Hq + Hkv) * D], d[:, (Hq + Hkv) * D :], B, S, Hq,
                        Hkv, D, causal=causal, rope=rope)
        grads.append(d if rope is not None else K.rope_(d, table, S, Hq + Hkv, D, backward=True))
    K.check_status(out.device)
    a, b = (g.float() for g in grads)
    assert (a - b).norm() < 2**-8 * a.norm() and torch.equal(grads[0][:, (Hq + Hkv) * D :], grads[1][:, (Hq + Hkv) * D :])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("S,Hq,Hkv", [(1, 2, 1), (129, 3, 1), (256, 7, 1), (300, 12, 2), (1000, 8, 2), (1280, 6, 1)])
def test_attention_bwd_shares_heads(S, Hq, Hkv, causal, D):
    """A batch that leaves SMs idle shares the heads of a group out, one beyond a block a SM does not: the same sums in another
    order in fp32 (far below a rounding to bf16, which may then fall to the other side: 2^-8 of the value)."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B = sms // ((S + 127) // 128 * Hkv) + 1
    qkv, q, k, v = _qkv(B, S, Hq, Hkv, D, seed=S + D)
    table = K.rope_table(S, D, 10000.0, "cuda")
    out = torch.empty(B * S, Hq * D, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device="cuda")
    K.attention_fwd(q, k, v, B, S, Hq, Hkv, D, out, lse, causal=causal, any_length=True)
    d_o = torch.randn_like(out)
    a, b = Hq * D, (Hq + Hkv) * D
    grads = []
    for n in (B, 1):
        d = torch.full_like(qkv, 7.0)
        K.attention_bwd(q, k, v, out, d_o, lse, d[:, :a], d[:, a:b], d[:, b:], n, S, Hq, Hkv, D, causal=causal, rope=table,
                        any_length=True)
        grads.append(d[:S].float())
        assert bool((d[n * S :] == 7).all())
    K.check_status(out.device)
    for lo, hi in ((0, a), (a, b), (b, qkv.shape[1])):
        assert (grads[0][:, lo:hi] - grads[1][:, lo:hi]).norm() <= 2**-8 * grads[0][:, lo:hi].norm() + 1e-6 * d_o.float()[:S].norm()


@pytest.mark.parametrize("D,poly", [(64, None), (64, "0"), (64, "4"), (128, "0"), (128, "4")])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("key", [*range(8), 131, 200])
def test_attention_fwd_keeps_non_finite_scores(monkeypatch, D, poly, bad, key):
    """A key with a NaN or an infinity spoils the rows that see it, whichever unit its exponentials are computed on
    (`poly` of every eight on the FMA pipe, None: the default), and no others."""
    B, S, Hq, Hkv = 1, 256, 2, 1
    monkeypatch.setenv("FTB200_ATTN_FWD", "pair")
    if poly is None:
        monkeypatch.delenv("FTB200_ATTN_POLY", raising=False)
    else:
        monkeypatch.setenv("FTB200_ATTN_POLY", poly)
    _, q, k, v = _qkv(B, S, Hq, Hkv, D, seed=key)
    k[key, 0] = bad
    out = torch.empty(B * S, Hq * D, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, Hq, S, dtype=torch.float32, device="cuda")
    K.attention_fwd(q, k, v, B, S, Hq, Hkv, D, out, lse)
    K.check_status(out.device)
    q4, k4, v4 = (t.reshape(B, S, -1, D) for t in (q, k, v))
    ref = K.ref_attention(q4.float(), k4.float(), v4.float(), True)
    got = out.float().reshape(ref.shape)
    fine = ref.isfinite().all(-1)
    assert torch.equal(got.isfinite().all(-1), fine) and not got[~fine].isfinite().any()
    assert torch.equal(lse.isfinite(), fine.transpose(1, 2)) and (~fine).sum() >= (S - key) // 2
    assert (got[fine] - ref[fine]).norm() <= 1e-2 * ref[fine].norm()  # no row is left where the first key is NaN


@pytest.mark.parametrize("D,poly", [(64, None), (64, "4"), (128, "4")])
@pytest.mark.parametrize("first", [97, 128, 230])
def test_attention_fwd_masked_keys_have_no_weight(monkeypatch, D, poly, first):
    """Values behind the mask, however large, leave the rows before them bit for bit as they are: the weight of a masked
    score is zero on either unit."""
    B, S, Hq, Hkv = 1, 256, 2, 1
    monkeypatch.setenv("FTB200_ATTN_FWD", "pair")
    if poly is None:
        monkeypatch.delenv("FTB200_ATTN_POLY", raising=False)
    else:
        monkeypatch.setenv("FTB200_ATTN_POLY", poly)
    _, q, k, v = _qkv(B, S, Hq, Hkv, D, seed=first)
    outs = []
    for big in (0.0, 3e38):
        v[first:] = big
        out = torch.empty(B * S, Hq * D, dtype=torch.bfloat16, device="cuda")
        K.attention_fwd(q, k, v, B, S, Hq, Hkv, D, out)
        K.check_status(out.device)
        outs.append(out[:first])
    assert torch.equal(*outs)
