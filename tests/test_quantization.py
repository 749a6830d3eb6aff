"""fp8 block quantisation: format round trip, kernels against the PyTorch restatement,
quantised collectives over gloo (CPU) and the fused peer kernel (GPU, emulated team).
Error bounds follow the thresholds the reference asserts (mean relative error <= 0.05)."""
import ctypes
from concurrent.futures import ThreadPoolExecutor
from datetime import timedelta

import pytest
import torch
import torch.distributed as dist
from torch.distributed.distributed_c10d import ReduceOp

from torchft_b200 import quantization as Q
from torchft_b200.collectives import allreduce_quantized, reduce_scatter_quantized, allocate_reduce_scatter_output
from torchft_b200.ops import _native as N
from torchft_b200.process_group import ProcessGroupGloo


def mean_rel_err(a, b):
    a, b = a.float(), b.float()
    return ((a - b).abs().mean() / b.abs().mean()).item()


def with_outliers(n, seed, mult=100.0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(n, generator=g)
    idx = torch.randperm(n, generator=g)[: max(1, n // 1000)]
    x[idx] *= mult
    return x


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [128, 4096, 128 * 1000])
def test_roundtrip_cpu(dtype, n):
    x = with_outliers(n, 0).to(dtype)
    buf = torch.empty(Q.quantized_nbytes(n), dtype=torch.uint8)
    Q.quantize_into(x, buf)
    y = torch.empty_like(x)
    Q.dequantize_from(buf, y)
    assert mean_rel_err(y, x) < 0.05
    # a block of zeros stays zero and has a finite scale
    z = torch.zeros(256, dtype=dtype)
    zb = torch.empty(Q.quantized_nbytes(256), dtype=torch.uint8)
    Q.quantize_into(z, zb)
    out = torch.ones(256, dtype=dtype)
    Q.dequantize_from(zb, out)
    assert out.abs().sum() == 0


def test_list_api_and_padding_cpu():
    ts = [torch.randn(5, 7), torch.randn(130), torch.randn(3, 3, 3)]
    orig = [t.clone() for t in ts]
    buf, (n,) = Q.fused_quantize_into_fp8(ts, world_size=3)
    assert n % (128 * 3) == 0 and buf.numel() == Q.quantized_nbytes(n)
    for t in ts:
        t.zero_()
    Q.fused_dequantize_from_fp8(ts, buf, world_size=3)
    for t, o in zip(ts, orig):
        assert mean_rel_err(t, o) < 0.06


def _gloo(world):
    store = dist.TCPStore("localhost", 0, is_master=True, wait_for_workers=False)
    pgs = [ProcessGroupGloo(timeout=timedelta(seconds=20)) for _ in range(world)]
    with ThreadPoolExecutor(max_workers=world) as ex:
        list(ex.map(lambda r: pgs[r].configure(f"localhost:{store.port}/q", "r", r, world), range(world)))
    for r, pg in enumerate(pgs):
        pg._rank = r
    return store, pgs


@pytest.mark.parametrize("op", [ReduceOp.SUM, ReduceOp.AVG])
def test_allreduce_quantized_gloo(op):
    world = 2
    store, pgs = _gloo(world)
    try:
        data = [[with_outliers(1000, 10 * r + i).reshape(10, 100) for i in range(2)] for r in range(world)]
        want = [sum(data[r][i] for r in range(world)) / (world if op == ReduceOp.AVG else 1) for i in range(2)]

        def run(r):
            ts = [t.clone() for t in data[r]]
            allreduce_quantized(ts, op, pgs[r]).wait()
            return ts

        with ThreadPoolExecutor(max_workers=world) as ex:
            outs = list(ex.map(run, range(world)))
        for ts in outs:
            for t, w in zip(ts, want):
                assert mean_rel_err(t, w) < 0.05
        for a, b in zip(outs[0], outs[1]):
            assert torch.equal(a, b)  # every rank ends with identical values
    finally:
        for pg in pgs:
            pg.shutdown()


def test_reduce_scatter_quantized_gloo():
    world = 2
    store, pgs = _gloo(world)
    try:
        data = [[with_outliers(1024, 3 * r)] for r in range(world)]
        total = (data[0][0] + data[1][0])

        def run(r):
            out, n = allocate_reduce_scatter_output(data[r], world)
            reduce_scatter_quantized(out, [t.clone() for t in data[r]], ReduceOp.SUM, pgs[r]).wait()
            return out

        with ThreadPoolExecutor(max_workers=world) as ex:
            outs = list(ex.map(run, range(world)))
        per = 1024 // world
        for r, o in enumerate(outs):
            assert mean_rel_err(o, total[r * per : (r + 1) * per]) < 0.05
    finally:
        for pg in pgs:
            pg.shutdown()


def _factorisations(n):
    return [(a, n // a) for a in range(1, n + 1) if n % a == 0]


def _simulated_allreduce(per_rank, scale):
    """The quantised allreduce for ranks that live in one process: quantise each rank's flat data, hand slice r of
    every rank to rank r, reduce there, gather the reduced slices, dequantise (the data flow of allreduce_quantized
    with the collectives replaced by slicing)."""
    ws = len(per_rank)
    n = Q.padded_numel(per_rank[0].numel(), ws)
    per = n // ws
    qbufs = []
    for x in per_rank:
        flat = torch.zeros(n, dtype=x.dtype)
        flat[: x.numel()] = x.reshape(-1)
        b = torch.empty(Q.quantized_nbytes(n), dtype=torch.uint8)
        Q.quantize_into(flat, b)
        qbufs.append(b)
    full = torch.empty(Q.quantized_nbytes(n), dtype=torch.uint8)
    fc, fs = Q.split_quantized(full, n)
    nb = per // Q.BLOCK
    for r in range(ws):
        parts = []
        for k in range(ws):
            c, sc = Q.split_quantized(qbufs[(r + k) % ws], n)
            b = torch.empty(Q.quantized_nbytes(per), dtype=torch.uint8)
            bc, bs = Q.split_quantized(b, per)
            bc.copy_(c[r * per : (r + 1) * per])
            bs.copy_(sc[r * nb : (r + 1) * nb])
            parts.append(b)
        red = torch.empty(Q.quantized_nbytes(per), dtype=torch.uint8)
        Q.reduce_quantized(parts, per, scale, red)
        rc, rs = Q.split_quantized(red, per)
        fc[r * per : (r + 1) * per].copy_(rc)
        fs[r * nb : (r + 1) * nb].copy_(rs)
    out = torch.empty(n, dtype=per_rank[0].dtype)
    Q.dequantize_from(full, out)
    return out[: per_rank[0].numel()]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("avg", [False, True])
def test_simulated_two_rank_allreduce_matrix(dtype, avg):
    """Sizes x multipliers x every 2-D factorisation of the size, two simulated ranks, against the exact
    reduction; mean relative error <= 0.05 (the matrix of torchft/quantization_test.py:35-131)."""
    ws = 2
    g = torch.Generator().manual_seed(5)
    for size in (128, 512, 4096):
        for mult in (1.0, 100.0, 1000.0):
            if dtype == torch.float16 and mult == 1000.0 and not avg:
                mult = 500.0  # keep the exact sum inside fp16's range
            for rows, cols in _factorisations(size):
                xs = [(torch.rand(rows, cols, generator=g) * mult).to(dtype) for _ in range(ws)]
                want = sum(x.float() for x in xs) * (1.0 / ws if avg else 1.0)
                got = _simulated_allreduce(xs, 1.0 / ws if avg else 1.0).view(rows, cols)
                assert got.dtype == dtype
                assert mean_rel_err(got, want) <= 0.05, (size, mult, rows, cols)


# ------------------------------------------------------------------------------------ GPU


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_kernels_match_reference_gpu(dtype):
    n = 128 * 4099
    x = with_outliers(n, 1).to(dtype).cuda()
    sub = with_outliers(n, 2).to(dtype).cuda()
    buf = torch.empty(Q.quantized_nbytes(n), dtype=torch.uint8, device="cuda")
    Q.quantize_into(x, buf)
    codes, scales = Q.split_quantized(buf, n)
    rc, rs = Q.ref_quantize(x)
    torch.testing.assert_close(scales, rs, rtol=1e-6, atol=0)
    assert (codes != rc).float().mean().item() < 1e-3  # rounding ties may differ in a handful of codes
    y = torch.empty_like(x)
    Q.dequantize_from(buf, y)
    assert mean_rel_err(y, x) < 0.05
    Q.quantize_into(x, buf, minus=sub)  # fused pseudo-gradient
    Q.dequantize_from(buf, y)
    assert mean_rel_err(y, x.float() - sub.float()) < 0.05


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("numels", [
    [1], [128], [127, 1, 0, 129], [16] * 7, [5, 7, 11, 13, 4096, 3], [1] * 300,   # more tensors than one launch takes
    [128 * 1000 + 8, 64, 128 * 333], [100_003, 128 * 517, 40],
])
def test_list_kernels_match_flat_kernels_gpu(numels, dtype):
    """The list kernels give, bit for bit, what packing into a flat tensor and the flat kernels give, whatever the
    tensors' sizes, alignments and strides."""
    world = 3
    ts = [with_outliers(k, i).to(dtype).cuda() if k else torch.empty(0, dtype=dtype, device="cuda") for i, k in enumerate(numels)]
    ts.append(torch.randn(64, 48, device="cuda").to(dtype).t())           # not contiguous
    ts.append(torch.randn(1000, device="cuda").to(dtype)[1:])             # not on a 16-byte boundary
    n = Q.padded_numel(sum(t.numel() for t in ts), world)
    flat = torch.zeros(n, dtype=dtype, device="cuda")
    flat[: sum(t.numel() for t in ts)] = torch.cat([t.reshape(-1) for t in ts])
    want = torch.empty(Q.quantized_nbytes(n), dtype=torch.uint8, device="cuda")
    Q.quantize_into(flat, want)
    buf, (got_n,) = Q.fused_quantize_into_fp8(ts, world)
    assert got_n == n and torch.equal(buf, want)
    Q.dequantize_from(want, flat)
    versions = [t._version for t in ts]
    for t in ts:
        t.fill_(float("nan"))
    Q.fused_dequantize_from_fp8(ts, buf, world)
    assert torch.equal(torch.cat([t.reshape(-1) for t in ts]), flat[: sum(t.numel() for t in ts)])
    assert all(t._version > v for t, v in zip(ts, versions))
    leaf = torch.zeros(256, dtype=dtype, device="cuda", requires_grad=True)
    with pytest.raises(RuntimeError):  # as any write in place to a leaf
        Q.fused_dequantize_from_fp8([leaf], Q.fused_quantize_into_fp8([leaf], world)[0], world)


@pytest.mark.gpu
@pytest.mark.parametrize("head", [0, 1, 8, 2048, 2049])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_list_kernel_encodes_special_values_gpu(dtype, head):
    """Parts of 2048 elements that lie in one tensor are encoded from their packed values: the same bytes as the flat kernel
    gives, for NaN, infinities, negative zero, the smallest and largest numbers and blocks of zeros, whether the part begins
    on a 16-byte boundary, a tensor's end lies in it or not."""
    g = torch.Generator(device="cuda").manual_seed(head)
    x = torch.randn(3 * 2048 + 77, generator=g, device="cuda", dtype=dtype)
    x[:128] = 0.0
    x[130], x[300], x[301], x[500], x[700] = float("nan"), float("inf"), -float("inf"), -0.0, torch.finfo(dtype).tiny
    x[900], x[1100:1228], x[2100], x[5000] = torch.finfo(dtype).max, float("nan"), torch.finfo(dtype).tiny / 8, -torch.finfo(dtype).max
    lead = torch.randn(head, generator=g, device="cuda", dtype=dtype)
    ts = ([lead] if head else []) + [x]
    buf, (n,) = Q.fused_quantize_into_fp8(ts, 2)
    flat = torch.zeros(n, dtype=dtype, device="cuda")
    flat[: head + x.numel()] = torch.cat(ts)
    want = Q.quantize_into(flat, torch.empty_like(buf))
    assert torch.equal(buf, want)



def test_a_buffer_that_is_too_short_is_refused():
    """A buffer packed for fewer ranks (less padding), cut short, or of another type, before anything reads it."""
    ts = [torch.randn(1000), torch.randn(77)]
    buf, (n,) = Q.fused_quantize_into_fp8(ts, 2)
    for bad in (buf[:-1], buf[: n], buf.view(torch.int16), buf[None], buf[:0]):
        with pytest.raises(AssertionError):
            Q.fused_dequantize_from_fp8(ts, bad, 2)
        with pytest.raises(AssertionError):
            Q.dequantize_from(bad, torch.empty(n))
    with pytest.raises(AssertionError):
        Q.fused_dequantize_from_fp8(ts, buf, 16)
    Q.fused_dequantize_from_fp8(ts, buf.view(torch.int8), 2)  # bytes are bytes


@pytest.mark.parametrize("dtype,step", [(0, 8), (1, 4)])
def test_misaligned_codes_are_refused_before_the_launch(dtype, step):
    """The C entries look at the addresses (made up here) before they launch anything."""
    lib, n = N.lib(), 256
    bad_arg, align = -1, -2
    data, numel = (ctypes.c_void_p * 1)(1 << 20), (ctypes.c_longlong * 1)(n + 1)  # one element too many: refused as well

    def both(codes, scales, d=data):  # far apart: nothing shares memory
        return {fn(d, numel, ctypes.c_int(1), ctypes.c_void_p(codes), ctypes.c_void_p(scales), ctypes.c_longlong(n),
                   ctypes.c_int(dtype), ctypes.c_void_p(0)) for fn in (lib.ftb200_quantize_list_fp8, lib.ftb200_dequantize_list_fp8)}

    assert both(1 << 21, 1 << 22) == both((1 << 21) + step, 1 << 22) == {bad_arg}
    assert both((1 << 21) + step // 2, 1 << 22) == {align}
    assert both(1 << 21, (1 << 22) + 2) == {align}
    assert both(1 << 21, 1 << 22, (ctypes.c_void_p * 1)((1 << 20) + 1)) == {align}


@pytest.mark.gpu
def test_a_buffer_that_is_too_short_is_refused_gpu():
    ts = [torch.randn(1000, device="cuda")]
    buf, (n,) = Q.fused_quantize_into_fp8(ts, 2)
    with pytest.raises(AssertionError):
        Q.fused_dequantize_from_fp8(ts, buf[:-1], 2)
    with pytest.raises(AssertionError):
        Q.fused_dequantize_from_fp8(ts, buf, 16)
    out = [torch.empty_like(ts[0])]
    Q.fused_dequantize_from_fp8(out, buf.cpu(), 2)  # a buffer elsewhere comes over first
    Q.fused_dequantize_from_fp8(ts, buf, 2)
    assert torch.equal(out[0], ts[0])


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_tensors_without_storage_are_zeros(device):
    """Zeros as forward-mode autograd makes them have no memory to read, or to write."""
    x = torch.randn(300).to(device)
    zero = torch._efficientzerotensor((77,), device=device)
    got, _ = Q.fused_quantize_into_fp8([x, zero], 2)
    want, _ = Q.fused_quantize_into_fp8([x, torch.zeros(77, device=device)], 2)
    assert torch.equal(got, want)
    with pytest.raises(RuntimeError):
        Q.fused_dequantize_from_fp8([x, zero], got, 2)


def test_copies_that_overlap_a_direct_target_are_recognised():
    def overlap(*ts):
        return Q._copies_overlap(list(ts), [type(t) is torch.Tensor and t.is_contiguous() for t in ts])

    x, y = torch.zeros(1000), torch.zeros(64, 48)
    assert not overlap(x[:600], x[600:], y.t(), torch.zeros(0))
    assert not overlap(y[:, :16], x, y[:, 16:])            # interleaved, written by copies one after the other
    assert overlap(y.t(), x, y[63:]) and overlap(y[60:], y.t())
    assert overlap(x[::2], x[999:], y) is False and overlap(x[1::2], x[999:], y)
    assert overlap(x[100:500:2], x, y)                     # inside
    assert overlap(y[:, 1:].view(torch.uint8), y[:1].view(torch.uint8)[:, 8:].flatten()[:4])
    assert overlap(x, y.as_subclass(type("Sub", (torch.Tensor,), {})))


@pytest.mark.parametrize("dtype,size", [(0, 2), (1, 4)])
def test_targets_that_share_memory_are_refused_before_the_launch(dtype, size):
    """The C entry that writes a list looks at the addresses (made up here) before it launches anything; lists that pass
    are refused for the elements that they have too many."""
    lib, n, bad_arg, share = N.lib(), 256, -1, N.E_LIST
    codes, scales = 1 << 22, (1 << 22) + n

    def call(fn, *spans):
        data = (ctypes.c_void_p * len(spans))(*[a for a, _ in spans])
        numel = (ctypes.c_longlong * len(spans))(*[k for _, k in spans])
        return fn(data, numel, ctypes.c_int(len(spans)), ctypes.c_void_p(codes), ctypes.c_void_p(scales), ctypes.c_longlong(n),
                  ctypes.c_int(dtype), ctypes.c_void_p(0))

    def dq(*spans):
        return call(lib.ftb200_dequantize_list_fp8, *spans)

    a = 1 << 20
    assert dq((a, 200), (a + 200 * size, 200)) == dq((a + 200 * size, 200), (a, 200), (a + 100 * size, 0)) == bad_arg
    assert dq((a, 200), (a + 199 * size, 200)) == share     # one element in common
    assert dq((a, 10), (1 << 21, 300), (a, 10)) == share    # listed twice
    assert dq((a, 300), (a + 50 * size, 10)) == share       # inside
    assert dq((codes - 300 * size, 300)) == bad_arg and dq((codes - 299 * size, 300)) == share
    assert dq((scales + n // 128 * 4, 300)) == bad_arg and dq((scales + n // 128 * 4 - size, 300)) == share
    assert dq((a, 300), (0, 1)) == share and dq((a, 300), (0, 0)) == bad_arg
    assert call(lib.ftb200_quantize_list_fp8, (a, 200), (a, 200)) == bad_arg  # reading the same twice is fine


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_overlapping_targets_are_written_in_order_gpu(dtype):
    """Tensors that share memory end as copies in the list's order leave them: the last one wins."""
    base = with_outliers(5000, 3).to(dtype).cuda()

    def views(b):
        return [b[:1000], b[3000:4000].view(40, 25).t(), b[500:1700], b[:1000], b[3500:3777], b[2000:2001]]

    ts = views(base)
    buf, (n,) = Q.fused_quantize_into_fp8(ts, 2)
    flat = torch.empty(n, dtype=dtype, device="cuda")
    Q.dequantize_from(buf, flat)
    want, off = base.clone(), 0
    for t in views(want):
        t.copy_(flat[off : off + t.numel()].view_as(t))
        off += t.numel()
    Q.fused_dequantize_from_fp8(ts, buf, 2)
    assert torch.equal(base, want)


@pytest.mark.gpu
@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_fused_allreduce_fp8_emulated(world, dtype):
    from test_team_gpu import Emu
    from torchft_b200.ops import _native as N

    n = 128 * world * 37
    emu = Emu(world, Q.quantized_nbytes(n) + 256)
    arenas = [emu.arenas[r][emu.fb:] for r in range(world)]
    ins = [with_outliers(n, 100 + r).to(dtype).cuda() for r in range(world)]
    outs = [torch.empty(n, dtype=dtype, device="cuda") for _ in range(world)]
    want = sum(t.float() for t in ins) / world
    rc = emu.lib.ftb200_team_allreduce_fp8_emulated(
        emu.descs(), ctypes.c_int(world), emu.ptrs(arenas), emu.ptrs(ins), None, emu.ptrs(outs), ctypes.c_longlong(n),
        ctypes.c_int(0 if dtype == torch.bfloat16 else 1), ctypes.c_float(1.0 / world), ctypes.c_int(2), N.stream_ptr())
    assert rc == 0
    torch.cuda.synchronize()
    assert all(int(s.item()) == 0 for s in emu.status)
    for o in outs:
        assert torch.equal(o, outs[0])
        assert mean_rel_err(o, want) < 0.05


@pytest.mark.gpu
def test_diloco_outer_step_kernel_matches_torch_sgd_nesterov():
    from torchft_b200.ops.diloco import outer_step_

    torch.manual_seed(0)
    n = 4 * 1001
    backup = torch.randn(n, device="cuda")
    param = backup + 0.1 * torch.randn(n, device="cuda")
    ref_p = torch.nn.Parameter(backup.clone())
    opt = torch.optim.SGD([ref_p], lr=0.7, momentum=0.9, nesterov=True)
    mom = torch.zeros(n, device="cuda")
    for step in range(3):
        g = torch.randn(n, device="cuda")
        local = param.clone()
        outer_step_(g, mom, backup, param, lr=0.7, momentum_coef=0.9, alpha=0.25, nesterov=True, first_step=step == 0)
        ref_p.grad = g.clone()
        opt.step()
        torch.testing.assert_close(backup, ref_p.data, rtol=1e-5, atol=1e-6)
        torch.testing.assert_close(param, torch.lerp(ref_p.data, local, 0.25), rtol=1e-5, atol=1e-6)
        param = backup + 0.1 * torch.randn(n, device="cuda")
