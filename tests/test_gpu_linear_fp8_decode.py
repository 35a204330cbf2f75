"""GPU parity of the decode-width FP8-row projection (T <= 16, exact bf16 activations) through the C ABI.

Bars are the reference's own for its A16 path (tests/kernels/linear/test_linear.cpp:38-49,196-320):
against an fp64 dot product over the E4M3 weight values and the bf16 activations, times the row
scale, pushed through the epilogue in fp64,
  max(|got - ref| - allowance) <= 2e-3 * rms(ref), allowance = 1.001 * 2^-8 |ref| for bf16 outputs, 0 for fp32,
  and at least 99 % of the bf16 outputs equal bf16_rne(ref);
repeated calls are bitwise identical. The activation split that feeds the tensor core (three E5M2
pieces per value) is checked to be exact: scale * (p0 + p1 + p2) == x bit for bit."""
import numpy as np
import pytest

from fngine_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu
KTOL = 2e-3


def _torch():
    import torch
    assert torch.cuda.is_available()
    return torch


def bf16_tensor(torch, x):
    return torch.from_numpy(synth.to_bf16_bits(x).view(np.int16)).cuda().view(torch.bfloat16)


def make_weight(torch, seed, n, k, bf16_scales):
    from fngine_b200 import linear
    codes, scales = synth.fp8_row_weight(seed, n, k)
    wc, ws = torch.from_numpy(codes).cuda(), torch.from_numpy(scales).cuda()
    if bf16_scales:
        ws = ws.to(torch.bfloat16)
    return linear.Fp8RowWeight(wc, ws)


def exact_acc(torch, x, weight):
    """fp64 [T][n]: (x . W^T) * scale over the represented values."""
    tab = torch.from_numpy(O.e4m3_table().astype(np.float64)).cuda()
    out = torch.empty(x.shape[0], weight.n, dtype=torch.float64, device="cuda")
    xd = x.double()
    for r0 in range(0, weight.n, 4096):  # bounded fp64 temporaries
        w = tab[weight.codes[r0:r0 + 4096].long()]
        out[:, r0:r0 + 4096] = (xd @ w.T) * weight.scales[r0:r0 + 4096].double()[None, :]
    return out


def compare(torch, got, ref, bf16_out):
    got, ref = got.double().reshape(-1), ref.reshape(-1)
    rms = float(ref.pow(2).mean().sqrt())
    allowance = ref.abs() * (2.0 ** -8 * 1.001) if bf16_out else 0.0
    worst = float(((got - ref).abs() - allowance).max())
    assert bool(torch.isfinite(got).all())
    assert worst <= KTOL * rms, (worst, rms)
    if bf16_out:
        match = float((got.float() == ref.float().to(torch.bfloat16).float()).double().mean())
        assert match >= 0.99, match
        return worst / rms, match
    return worst / rms, 1.0


CASES = [
    # T, n, k, epilogue, bf16 row scales
    (1, 1280, 2560, "swiglu", True),          # moe.shared_gate_up
    (16, 1280, 2560, "swiglu", False),
    (9, 2560, 640, "shared_scale", True),     # moe.shared_down: five K blocks, every tile is shared by CTAs
    (5, 2560, 6144, "gr_write", True),        # gdn.out / qsa.o
    (16, 16384, 2560, "store_bf16", True),    # gdn.qkvz
    (3, 320, 10240, "store_f32", False),      # three row tiles, eighty K blocks each
    (7, 1000, 384, "store_bf16", False),      # ragged last row tile
    (16, 24832, 2560, "store_f32", True),     # a tenth of the vocabulary projection
    (2, 208, 256, "swiglu", False),           # 104 gate rows: ragged 64-row halves
    (4, 128, 128, "store_f32", True),         # one tile, one K block, one CTA
]


@pytest.mark.parametrize("T,n,k,kind,bf16_scales", CASES)
def test_linear_fp8_decode_matches_the_exact_product(T, n, k, kind, bf16_scales):
    torch = _torch()
    from fngine_b200 import linear
    weight = make_weight(torch, 300 + n + T, n, k, bf16_scales)
    x = bf16_tensor(torch, synth.activations(500 + T + k, T, hidden=k) * np.float32(1.7))
    work = linear.linear_fp8_decode_workspace(weight)
    acc = exact_acc(torch, x, weight)
    gen = torch.Generator(device="cpu").manual_seed(7 + T)
    if kind == "store_bf16":
        out = torch.full((T, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        make = lambda o: linear.store_bf16(o)
        ref, bf16_out = acc, True
    elif kind == "store_f32":
        out = torch.full((T, n), float("nan"), dtype=torch.float32, device="cuda")
        make = lambda o: linear.store_f32(o)
        ref, bf16_out = acc, False
    elif kind == "swiglu":
        out = torch.full((T, n // 2), float("nan"), dtype=torch.bfloat16, device="cuda")
        make = lambda o: linear.swiglu(o)
        g, u = acc[:, :n // 2], acc[:, n // 2:]
        ref, bf16_out = g / (1.0 + torch.exp(-g)) * u, True
    elif kind == "shared_scale":
        logits = torch.randn(T, 513, generator=gen).cuda()
        out = torch.full((T, n), float("nan"), dtype=torch.float32, device="cuda")
        make = lambda o: linear.shared_scale(o, logits[:, 512:], 513)
        ref, bf16_out = acc * torch.sigmoid(logits[:, 512].double())[:, None], False
    else:
        inj = torch.randn(T, 4, generator=gen).cuda()
        x0 = torch.randn(T, 4, n, generator=gen).cuda()
        out = x0.clone()
        make = lambda o: linear.gr_write(o, inj)
        ref, bf16_out = inj.double()[:, :, None] * acc[:, None, :], False
    linear.linear_fp8_decode(x, weight, make(out), work)
    torch.cuda.synchronize()
    got = out.double() - x0.double() if kind == "gr_write" else out
    ratio, match = compare(torch, got, ref, bf16_out)
    print("fp8 decode T=%d %dx%d %s: worst excess / rms %.2e, bf16 rounding match %.4f" % (T, n, k, kind, ratio, match))
    # deterministic: a second call (fresh output) is bitwise identical
    out2 = x0.clone() if kind == "gr_write" else torch.empty_like(out)
    linear.linear_fp8_decode(x, weight, make(out2), work)
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int16 if out.dtype == torch.bfloat16 else torch.int32),
                       out2.view(torch.int16 if out.dtype == torch.bfloat16 else torch.int32))


def test_activation_pieces_are_exact():
    """scale[t] * (p0 + p1 + p2) reproduces the bf16 activations bit for bit over a 2^23 dynamic range
    inside a row; an all-zero token, a tiny token, and unused token slots left as zero rows. The pieces of the streaming
    kernel, which more row tiles than multiprocessors take: they can be read back from the workspace."""
    torch = _torch()
    from fngine_b200 import linear
    T, n, k = 6, 19080, 1024
    weight = make_weight(torch, 11, n, k, False)
    x = synth.activations(99, T, hidden=k) * np.exp2(np.linspace(-12, 4, k, dtype=np.float32))[None, :]
    x[2] = 0.0
    x[4] *= np.float32(1e-6)
    xb = bf16_tensor(torch, x)
    work = linear.linear_fp8_decode_workspace(weight)
    out = torch.empty(T, n, dtype=torch.float32, device="cuda")
    linear.linear_fp8_decode(xb, weight, linear.store_f32(out), work)
    torch.cuda.synchronize()
    raw = work.cpu().numpy()
    pieces = raw[:48 * k].reshape(3, 16, k)
    scales = raw[48 * k:48 * k + 64].view(np.float32)
    vals = (pieces.astype(np.uint16) << 8).view(np.float16).astype(np.float64)  # E5M2 = the top byte of binary16
    want = xb.float().cpu().numpy().astype(np.float64)
    got = vals.sum(axis=0)[:T] * scales[:T, None].astype(np.float64)
    # exact wherever the value's last mantissa bit is at least 2^-16 of the scaled range (guaranteed for
    # |x| >= 2^-23 of the row maximum); below that the dropped bits are under 2^-30 of the row maximum
    rowmax = np.abs(want).max(axis=1, keepdims=True)
    err = np.abs(got - want)
    assert np.all((err == 0) | (np.abs(want) < rowmax * 2.0 ** -23))
    assert np.all(err <= rowmax * 2.0 ** -30)
    assert (err == 0).mean() > 0.99
    assert not pieces[:, T:].any()
    assert np.all(np.log2(scales[[0, 1, 3, 4, 5]]) == np.round(np.log2(scales[[0, 1, 3, 4, 5]])))  # powers of two


@pytest.mark.parametrize("T,n,k", [(1, 24832, 1024), (9, 19080, 2560)])
def test_projection_right_behind_the_kernel_that_wrote_its_weights(T, n, k):
    """More row tiles than multiprocessors, whose kernel asks for weight codes ahead of its own wait: codes copied in by
    the call before on the same stream, no synchronization between, give the bits of synchronized calls."""
    torch = _torch()
    from fngine_b200 import linear
    weights = [make_weight(torch, 40 + i, n, k, False) for i in range(2)]
    x = bf16_tensor(torch, synth.activations(700 + T, T, hidden=k))
    work = linear.linear_fp8_decode_workspace(weights[0])
    want = [torch.empty(T, n, dtype=torch.float32, device="cuda") for _ in weights]
    for w, o in zip(weights, want):
        linear.linear_fp8_decode(x, w, linear.store_f32(o), work)
        torch.cuda.synchronize()
    live = linear.Fp8RowWeight(weights[0].codes.clone(), weights[0].scales.clone())
    outs = [torch.empty_like(want[0]) for _ in range(12)]
    for i, o in enumerate(outs):
        live.codes.copy_(weights[i % 2].codes)
        live.scales.copy_(weights[i % 2].scales)
        live.codes[-1:].copy_(weights[i % 2].codes[-1:])  # (the last kernel ahead of the projection writes codes)
        linear.linear_fp8_decode(x, live, linear.store_f32(o), work)
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        assert torch.equal(o, want[i % 2]), i


@pytest.mark.parametrize("T", [1, 5, 16])
def test_projection_reads_what_the_kernel_ahead_of_it_wrote(T):
    """A projection whose activations the projection before it writes, chained in a CUDA graph and replayed on changing
    inputs: the bits of synchronized calls every time."""
    torch = _torch()
    from fngine_b200 import linear
    gu, dn = make_weight(torch, 61, 1280, 2560, True), make_weight(torch, 62, 2560, 640, True)
    works = [linear.linear_fp8_decode_workspace(w) for w in (gu, dn)]
    x = torch.empty(T, 2560, dtype=torch.bfloat16, device="cuda")
    h = torch.empty(T, 640, dtype=torch.bfloat16, device="cuda")
    y = torch.empty(T, 2560, dtype=torch.float32, device="cuda")
    inputs = [bf16_tensor(torch, synth.activations(900 + i, T, hidden=2560) * np.float32(2.0 ** (3 * (i % 3)))) for i in range(16)]
    epis = linear.swiglu(h), linear.store_f32(y)
    want = []
    for v in inputs:
        x.copy_(v)
        torch.cuda.synchronize()
        for src, w, e, k in zip((x, h), (gu, dn), epis, works):
            linear.linear_fp8_decode(src, w, e, k)
            torch.cuda.synchronize()
        want.append(y.clone())
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side):
        for src, w, e, k in zip((x, h), (gu, dn), epis, works):
            linear.linear_fp8_decode(src, w, e, k)
    for turn in range(4):
        got = []
        for v in inputs:
            x.copy_(v)
            graph.replay()
            got.append(y.clone())
        torch.cuda.synchronize()
        for i, g in enumerate(got):
            assert torch.equal(g, want[i]), (turn, i)


@pytest.mark.parametrize("T,n,k,kind", [(1, 2560, 2560, "store_bf16"), (16, 2560, 2560, "store_bf16"), (7, 1280, 2560, "store_f32"),
                                        (4, 512, 2560, "swiglu")])
def test_projection_into_the_memory_of_its_activations(T, n, k, kind):
    """The activations are read before anything is written: an output that starts inside them holds the product."""
    torch = _torch()
    from fngine_b200 import linear
    weight = make_weight(torch, 88, n, k, True)
    x = bf16_tensor(torch, synth.activations(31 + T, T, hidden=k))
    work = linear.linear_fp8_decode_workspace(weight)
    make = {"store_bf16": linear.store_bf16, "store_f32": linear.store_f32, "swiglu": linear.swiglu}[kind]
    shape, dt = (T, n // 2 if kind == "swiglu" else n), torch.float32 if kind == "store_f32" else torch.bfloat16
    values, ref = shape[0] * shape[1], exact_acc(torch, x, weight)
    if kind == "swiglu":
        ref = ref[:, :n // 2] / (1.0 + torch.exp(-ref[:, :n // 2])) * ref[:, n // 2:]
    for first in (0, 16 * (x.numel() // 32)):  # the output at the start of the activations, and from their middle on
        room = torch.empty(x.numel() + 16 + 2 * values, dtype=torch.bfloat16, device="cuda")
        xin = room[:x.numel()].view(T, k)
        xin.copy_(x)
        out = room[first:first + values * dt.itemsize // 2].view(dt).view(shape)
        linear.linear_fp8_decode(xin, weight, make(out), work)
        torch.cuda.synchronize()
        compare(torch, out, ref, dt == torch.bfloat16)


@pytest.mark.parametrize("T,n,k", [(6, 1024, 1024),     # eight row tiles, clusters of eight CTAs with one K block each
                                   (16, 2560, 2560),    # twenty row tiles, twenty K blocks: uneven shares
                                   (1, 8192, 1024),     # sixty-four row tiles: two CTAs each
                                   (9, 8, 10240),       # one ragged row tile, ten K blocks per CTA
                                   (5, 256, 640)])      # two row tiles, clusters of five
def test_activations_reach_the_sums_exactly(T, n, k):
    """The cluster kernel's own activation split, through its outputs: weight rows with a single 1 make each output one
    activation, bit for bit over a 2^23 dynamic range inside a row (below that to 2^-30 of the row's maximum, as above);
    an all-zero token, a tiny token."""
    torch = _torch()
    from fngine_b200 import linear
    at = torch.arange(n) % k if n >= k else torch.randperm(k, generator=torch.Generator().manual_seed(n))[:n]
    codes = torch.zeros(n, k, dtype=torch.uint8)
    codes[torch.arange(n), at] = 0x38  # E4M3 1.0
    weight = linear.Fp8RowWeight(codes.cuda(), torch.ones(n, dtype=torch.float32, device="cuda"))
    x = synth.activations(99, T, hidden=k) * np.exp2(np.linspace(-12, 4, k, dtype=np.float32))[None, :]
    if T > 4:
        x[2] = 0.0
        x[4] *= np.float32(1e-6)
    xb = bf16_tensor(torch, x)
    out = torch.full((T, n), float("nan"), dtype=torch.float32, device="cuda")
    linear.linear_fp8_decode(xb, weight, linear.store_f32(out), linear.linear_fp8_decode_workspace(weight))
    torch.cuda.synchronize()
    rows = xb.float().cpu().numpy().astype(np.float64)
    want, got = rows[:, at.numpy()], out.cpu().numpy().astype(np.float64)
    rowmax = np.abs(rows).max(axis=1, keepdims=True)
    err = np.abs(got - want)
    assert np.all((err == 0) | (np.abs(want) < rowmax * 2.0 ** -23))
    assert np.all(err <= rowmax * 2.0 ** -30)
    assert (err == 0).mean() > 0.99


@pytest.mark.parametrize("T", [4, 15])
def test_distance_of_a_shared_sum_from_the_exact_product(T):
    """Five partial tiles, one per CTA, and the shared-gate factor (2560 x 640): in relative L2 not further from the fp64
    product than the 7.0e-8 of a kernel that adds two or three partial tiles of two K blocks each. (Added one by one in
    fp32, with a reciprocal and two products behind, 7.1e-8 to 7.3e-8.)"""
    torch = _torch()
    from fngine_b200 import linear
    num = den = 0.0
    for seed in range(8):
        weight = make_weight(torch, 8800 + seed, 2560, 640, True)
        x = bf16_tensor(torch, synth.activations(8900 + seed + T, T, hidden=640))
        gate = torch.randn(T, 513, generator=torch.Generator().manual_seed(seed)).cuda()
        out = torch.empty(T, 2560, dtype=torch.float32, device="cuda")
        work = linear.linear_fp8_decode_workspace(weight)
        linear.linear_fp8_decode(x, weight, linear.shared_scale(out, gate[:, 512:], 513), work)
        torch.cuda.synchronize()
        ref = exact_acc(torch, x, weight) * torch.sigmoid(gate[:, 512].double())[:, None]
        num, den = num + float((out.double() - ref).norm()) ** 2, den + float(ref.norm()) ** 2
    print("distance %.3e" % (num / den) ** 0.5)
    assert (num / den) ** 0.5 <= 7.0e-8


def test_linear_fp8_decode_argument_errors():
    torch = _torch()
    import ctypes

    from fngine_b200 import lib as fblib
    lib = fblib.load()
    buf = torch.zeros(8 << 20, dtype=torch.uint8, device="cuda")
    p = buf.data_ptr()
    epi = fblib.LinearEpilogue(fblib.EPI_STORE_BF16, 0, p, None, None)
    e = ctypes.byref(epi)
    assert lib.fb_linear_fp8_decode(p, 17, p, p, 0, 256, 256, e, p, 8 << 20, None) == 1   # more than 16 tokens
    assert lib.fb_linear_fp8_decode(p, 4, p, p, 0, 256, 100, e, p, 8 << 20, None) == 1    # k % 128
    assert lib.fb_linear_fp8_decode(p, 4, p, p, 0, 256, 256, e, p, 1024, None) == 1       # workspace too small
    assert b"workspace" in lib.fb_last_error_string()
    bad = fblib.LinearEpilogue(fblib.EPI_GR_WRITE, 0, p, None, None)
    assert lib.fb_linear_fp8_decode(p, 4, p, p, 0, 256, 256, ctypes.byref(bad), p, 8 << 20, None) == 1  # no inj
    bad = fblib.LinearEpilogue(9, 0, p, None, None)
    assert lib.fb_linear_fp8_decode(p, 4, p, p, 0, 256, 256, ctypes.byref(bad), p, 8 << 20, None) == 1  # bad kind
