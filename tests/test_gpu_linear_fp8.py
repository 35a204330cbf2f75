"""GPU parity of the FP8-row dense projection above decode width (tcgen05 E4M3 GEMM) through the C ABI.

Two routes, as in the reference (src/kernels/linear/linear.h:27-37):

* exact (Auto / A16, the default): the bf16 activations are kept. Bar = the reference's own for its A16
  path (tests/kernels/linear/test_linear.cpp:8-11,38-49): against an fp64 product of the E4M3 weight
  values with the UNQUANTIZED bf16 activations, times the row scale, pushed through the epilogue,
  max(|got - ref| - allowance) <= 2e-3 rms(ref) with allowance = 1.001 * 2^-8 |ref| for bf16 outputs
  and 0 for fp32 outputs, and >= 99 % of bf16 outputs equal bf16_rne(ref). The benchmark shape is also
  held to the relative-L2 bar of 2e-2 against the fp32 reference on dequantized weights.
* A8 (on request): one E4M3 code per activation. Bar = the reference's for that path: the same rule
  against an oracle that applies the SAME per-token E4M3 quantization; its distance from the unquantized
  reference is mantissa-bound (about 2.6e-2 relative L2 for N(0,1) inputs, above the 2e-2 the exact
  route meets) and is only reported.
"""
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


def exact_acc(torch, a, weight):
    """fp64 [T][n]: (a . W^T) * scale over the represented values; a fp64 [T][k]."""
    tab = torch.from_numpy(O.e4m3_table().astype(np.float64)).cuda()
    out = torch.empty(a.shape[0], weight.n, dtype=torch.float64, device="cuda")
    for r0 in range(0, weight.n, 2048):  # bounded fp64 temporaries
        w = tab[weight.codes[r0:r0 + 2048].long()]
        out[:, r0:r0 + 2048] = (a @ w.T) * weight.scales[r0:r0 + 2048].double()[None, :]
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
    return worst / rms


def test_fp8_token_quantizer_bit_exact():
    torch = _torch()
    from fngine_b200 import linear
    x = synth.activations(61, 48) * np.linspace(0.01, 30, 48, dtype=np.float32)[:, None]
    x[5] = 0.0  # an all-zero token: scale 0, codes 0
    xb = synth.to_bf16_bits(x)
    codes, scales = linear.fp8_quantize_tokens(torch.from_numpy(xb.view(np.int16)).cuda().view(torch.bfloat16))
    want_c, want_s = O.quantize_tokens_e4m3(xb)
    assert np.array_equal(codes.cpu().numpy(), want_c)
    assert np.array_equal(scales.cpu().numpy().view(np.uint32), want_s.view(np.uint32))


def test_two_piece_split_is_bit_exact_and_lossless():
    """The exact route's activation pieces: bit-identical to the host statement, and scale * (hi + lo)
    gives the bf16 activation back - exactly for every element of at least 2^-9 of its row's scaled
    range (|v| >= 0.25 with the row maximum in [128, 256)), to 2^-10 of that range below."""
    torch = _torch()
    from fngine_b200 import linear
    x = synth.activations(62, 40) * np.logspace(-3, 3, 40, dtype=np.float32)[:, None]
    x[7] = 0.0
    x[9, :100] *= 1e-4  # tiny elements beside large ones
    xb = synth.to_bf16_bits(x)
    hi, lo, sc = linear.fp8_split_tokens(torch.from_numpy(xb.view(np.int16)).cuda().view(torch.bfloat16))
    w_hi, w_lo, w_sc = O.split_tokens_e4m3x2(xb)
    assert np.array_equal(hi.cpu().numpy(), w_hi) and np.array_equal(lo.cpu().numpy(), w_lo)
    assert np.array_equal(sc.cpu().numpy().view(np.uint32), w_sc.view(np.uint32))
    tab = O.e4m3_table().astype(np.float64)
    v = synth.bf16_bits_to_f32(xb).astype(np.float64)
    s = w_sc.astype(np.float64)[:, None]
    back = s * (tab[w_hi] + tab[w_lo])
    big = np.abs(v) >= 0.25 * s
    assert np.array_equal(back[big], v[big])
    assert np.all(np.abs(back - v) <= s * 2.0 ** -10)
    mx = np.abs(v).max(axis=1)
    live = mx > 0
    assert np.all((mx[live] / w_sc[live] >= 128) & (mx[live] / w_sc[live] < 256)) and np.all(w_sc[~live] == 0)


SHAPES = [(17, 256, 128, False), (64, 320, 640, True), (128, 1280, 2560, False), (300, 2560, 384, True),
          (512, 320, 256, False), (257, 192, 128, True)]


@pytest.mark.parametrize("T,N,K,bf16_scales", SHAPES)
def test_linear_fp8_exact_route(T, N, K, bf16_scales):
    """Auto (= exact activations) against the fp64 oracle on the unquantized bf16 activations."""
    torch = _torch()
    from fngine_b200 import linear
    weight = make_weight(torch, 900 + T, N, K, bf16_scales)
    x = bf16_tensor(torch, synth.activations(77 + T, T, hidden=K))
    out = torch.full((T, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    work = linear.linear_fp8_workspace(weight, T)
    linear.linear_fp8(x, weight, out, work)
    torch.cuda.synchronize()
    compare(torch, out, exact_acc(torch, x.double(), weight), True)
    out2 = torch.empty_like(out)
    linear.linear_fp8(x, weight, out2, work, path=linear.L.FP8_PATH_A16)  # A16 names the same route
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int16), out2.view(torch.int16))  # and repeated calls are bitwise identical


@pytest.mark.parametrize("T,N,K,bf16_scales", [(1, 256, 128, False), (3, 512, 256, False)] + SHAPES)
def test_linear_fp8_a8_route(T, N, K, bf16_scales):
    """A8 against the fp64 oracle fed the same per-token E4M3 activation quantization."""
    torch = _torch()
    from fngine_b200 import linear
    weight = make_weight(torch, 900 + T, N, K, bf16_scales)
    x = bf16_tensor(torch, synth.activations(77 + T, T, hidden=K))
    out = torch.full((T, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    work = linear.linear_fp8_workspace(weight, T)
    linear.linear_fp8(x, weight, out, work, path=linear.L.FP8_PATH_A8)
    torch.cuda.synchronize()
    xq, xs = linear.fp8_quantize_tokens(x)
    tab = torch.from_numpy(O.e4m3_table().astype(np.float64)).cuda()
    ref = exact_acc(torch, tab[xq.long()] * xs.double()[:, None], weight)
    got = out.double()
    rms = ref.pow(2).mean().sqrt()
    excess = ((got - ref).abs() - 2.0 ** -8 * ref.abs()).max()
    assert torch.isfinite(got).all()
    assert float(excess) <= KTOL * float(rms), (float(excess), float(rms))
    out2 = torch.empty_like(out)
    linear.linear_fp8(x, weight, out2, work, path=linear.L.FP8_PATH_A8)
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int16), out2.view(torch.int16))


@pytest.mark.parametrize("T", [24, 300])
@pytest.mark.parametrize("kind", ["store_f32", "gr_write", "swiglu", "shared_scale"])
def test_linear_fp8_epilogues_above_decode_width(T, kind):
    """The other epilogues of linear.h:64-103 on the GEMM path (the shapes the reference registers:
    gdn.out GrWrite 2560 x 6144, shared gate/up SwiGlu 1280 x 2560, shared down SharedScale 2560 x 640),
    exact route, against the fp64 oracle pushed through the same epilogue."""
    torch = _torch()
    from fngine_b200 import linear
    n, k = {"store_f32": (1024, 2560), "gr_write": (2560, 6144), "swiglu": (1280, 2560),
            "shared_scale": (2560, 640)}[kind]
    weight = make_weight(torch, 1300 + T, n, k, True)
    x = bf16_tensor(torch, synth.activations(88 + T, T, hidden=k))
    acc = exact_acc(torch, x.double(), weight)
    work = linear.linear_fp8_workspace(weight, T)
    g = torch.Generator(device="cuda").manual_seed(T)
    if kind == "store_f32":
        out = torch.full((T, n), float("nan"), dtype=torch.float32, device="cuda")
        epi, ref, bf = linear.store_f32(out), acc, False
    elif kind == "gr_write":
        inj = torch.randn(T, 4, device="cuda", generator=g)
        x0 = torch.randn(T, 4, n, device="cuda", generator=g)
        out = x0.clone()
        epi, bf = linear.gr_write(out, inj), False
        ref = x0.double() + inj.double()[:, :, None] * acc[:, None, :]
    elif kind == "swiglu":
        out = torch.full((T, n // 2), float("nan"), dtype=torch.bfloat16, device="cuda")
        gg, uu = acc[:, :n // 2], acc[:, n // 2:]
        epi, ref, bf = linear.swiglu(out), gg / (1.0 + torch.exp(-gg)) * uu, True
    else:
        logit = torch.randn(T, 513, device="cuda", generator=g)
        out = torch.full((T, n), float("nan"), dtype=torch.float32, device="cuda")
        epi, bf = linear.shared_scale(out, logit[:, 512:], 513), False
        ref = acc / (1.0 + torch.exp(-logit[:, 512].double()))[:, None]
    linear.linear_fp8(x, weight, epi, work)
    torch.cuda.synchronize()
    compare(torch, out, ref, bf)


def test_linear_fp8_on_a_weight_packed_by_the_reference_rule():
    """A bf16 weight matrix packed by the reference's FP8-row rule (tools/fp8row.py quantize_rows, restated in
    the oracle and pinned to the tool's own outputs: bf16 row scales, clamped round-to-nearest-even codes),
    then both routes against the fp64 product over the packed values; and the packing itself loses what
    E4M3 loses (about 3 % per element, 2.5e-2 relative L2 of the output), not more."""
    torch = _torch()
    from fngine_b200 import linear
    T, N, K = 96, 512, 1024
    wb = synth.to_bf16_bits((synth.normal(7001, N * K) * 0.02).astype(np.float32).reshape(N, K))
    wb[3] = 0  # an all-zero row: scale 0, codes 0
    codes, scales = O.quantize_fp8_rows(wb)
    weight = linear.Fp8RowWeight(torch.from_numpy(codes).cuda(),
                                 torch.from_numpy(scales.view(np.int16)).cuda().view(torch.bfloat16))
    x = bf16_tensor(torch, synth.activations(7002, T, hidden=K))
    out = torch.full((T, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    work = linear.linear_fp8_workspace(weight, T)
    linear.linear_fp8(x, weight, out, work)
    torch.cuda.synchronize()
    ref = exact_acc(torch, x.double(), weight)
    compare(torch, out, ref, True)
    assert float(out[:, 3].abs().max()) == 0.0
    dense = x.double() @ torch.from_numpy(synth.bf16_bits_to_f32(wb).astype(np.float64)).cuda().T
    assert float((ref - dense).norm() / dense.norm()) <= 4e-2


def test_linear_fp8_benchmark_shape():
    """bf16 [4096 x 2560] x E4M3 [9216 x 2560] with fp32 row scales -> bf16 [4096 x 9216], both routes.
    The stated bar (2e-2 relative L2 against an fp32 reference on dequantized weights and the given bf16
    activations) is asserted for the exact route, which is what Auto selects; for A8 the same figure is
    printed (mantissa-bound) and the GEMM is held to its own-quantization reference."""
    torch = _torch()
    from fngine_b200 import linear
    T, N, K = 4096, 9216, 2560
    weight = make_weight(torch, 4, N, K, False)
    wc, ws = weight.codes, weight.scales
    x = bf16_tensor(torch, synth.activations(44, T, hidden=K))
    out = torch.empty(T, N, dtype=torch.bfloat16, device="cuda")
    work = linear.linear_fp8_workspace(weight, T)
    tab = torch.from_numpy(O.e4m3_table()).cuda()
    wd = tab[wc.long()] * ws[:, None]                       # dequantized weights, fp32
    ref_u = x.float() @ wd.T                                # the given (unquantized) activations
    linear.linear_fp8(x, weight, out, work)
    torch.cuda.synchronize()
    rel_exact = float((out.float() - ref_u).norm() / ref_u.norm())
    linear.linear_fp8(x, weight, out, work, path=linear.L.FP8_PATH_A8)
    torch.cuda.synchronize()
    xq, xs = linear.fp8_quantize_tokens(x)
    ref_q = (tab[xq.long()] * xs[:, None]) @ wd.T           # same activation quantization
    got = out.float()
    rel_q = float((got - ref_q).norm() / ref_q.norm())
    rel_u = float((got - ref_u).norm() / ref_u.norm())
    print("fp8 gemm 4096x9216x2560: exact route rel L2 vs fp32 reference %.2e (bar 2e-2); A8 route %.2e vs its "
          "own-quantization reference, %.2e vs the fp32 reference" % (rel_exact, rel_q, rel_u))
    assert rel_exact <= 2e-2 and rel_exact <= 4e-3   # stated bar; bf16 output rounding alone is about 1.7e-3
    assert rel_q <= 4e-3
    assert rel_u <= 4e-2                              # A8's documented activation noise, not the stated bar


def test_linear_fp8_routes_decode_width_to_the_streaming_projection():
    """T <= 16 on the exact routes runs the decode-width projection: same bits as fb_linear_fp8_decode."""
    torch = _torch()
    from fngine_b200 import linear
    weight = make_weight(torch, 77, 1024, 512, True)
    x = bf16_tensor(torch, synth.activations(5, 9, hidden=512))
    a = torch.empty(9, 1024, dtype=torch.bfloat16, device="cuda")
    b = torch.empty_like(a)
    work = linear.linear_fp8_workspace(weight, 64)
    linear.linear_fp8(x, weight, a, work)
    linear.linear_fp8_decode(x, weight, linear.store_bf16(b), work)
    torch.cuda.synchronize()
    assert torch.equal(a.view(torch.int16), b.view(torch.int16))


def test_linear_fp8_argument_errors():
    torch = _torch()
    import ctypes
    from fngine_b200 import lib as fblib
    lib = fblib.load()
    buf = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    p = buf.data_ptr()
    epi = fblib.LinearEpilogue(fblib.EPI_STORE_BF16, 0, p, None, None)
    e = ctypes.byref(epi)
    assert lib.fb_linear_fp8(p, 32, p, p, 0, 100, 256, e, p, 1 << 20, None, 0) == 1   # n % 64
    assert lib.fb_linear_fp8(p, 32, p, p, 0, 128, 100, e, p, 1 << 20, None, 0) == 1   # k % 128
    assert lib.fb_linear_fp8(p, 32, p, p, 0, 128, 256, e, p, 16, None, 0) == 1        # workspace too small
    assert b"workspace" in lib.fb_last_error_string()
    assert lib.fb_linear_fp8(p, 32, p, p, 0, 128, 256, e, p, 1 << 20, None, 7) == 1   # unknown path
    sw = fblib.LinearEpilogue(fblib.EPI_SWIGLU, 0, p, None, None)
    assert lib.fb_linear_fp8(p, 32, p, p, 0, 192, 256, ctypes.byref(sw), p, 1 << 20, None, 0) == 1  # SwiGlu n % 128
    sh = fblib.LinearEpilogue(fblib.EPI_SHARED_SCALE, 513, p, None, None)
    assert lib.fb_linear_fp8(p, 32, p, p, 0, 128, 256, ctypes.byref(sh), p, 1 << 20, None, 0) == 1  # no gate logit


def epilogue_case(torch, kind, T, n, acc):
    """(maker of the epilogue with a fresh output, reference, whether bf16) over fp64 accumulators [T][n]."""
    from fngine_b200 import linear
    g = torch.Generator(device="cuda").manual_seed(T + n)
    nan = lambda w, dt: torch.full((T, w), float("nan"), dtype=dt, device="cuda")
    if kind == "store_bf16":
        return lambda: linear.store_bf16(nan(n, torch.bfloat16)), acc, True
    if kind == "store_f32":
        return lambda: linear.store_f32(nan(n, torch.float32)), acc, False
    if kind == "swiglu":
        gg, uu = acc[:, :n // 2], acc[:, n // 2:]
        return lambda: linear.swiglu(nan(n // 2, torch.bfloat16)), gg / (1.0 + torch.exp(-gg)) * uu, True
    if kind == "shared_scale":
        logit = torch.randn(T, 513, device="cuda", generator=g)
        return (lambda: linear.shared_scale(nan(n, torch.float32), logit[:, 512:], 513),
                acc * torch.sigmoid(logit[:, 512].double())[:, None], False)
    inj, x0 = torch.randn(T, 4, device="cuda", generator=g), torch.randn(T, 4, n, device="cuda", generator=g)
    return lambda: linear.gr_write(x0.clone(), inj), x0.double() + inj.double()[:, :, None] * acc[:, None, :], False


@pytest.mark.parametrize("path", ["auto", "a8"])
@pytest.mark.parametrize("T,n,k,kind", [
    (17, 64, 128, "store_f32"),        # smallest: half a row tile, one K block, one CTA
    (32, 128, 640, "swiglu"),          # one tile of 64 gate and 64 up rows, five K blocks over a cluster
    (33, 960, 384, "gr_write"),        # ragged rows, one token behind a multiple of 32, three K blocks
    (255, 2560, 896, "gr_write"),      # a token short of the two-SM kernel, seven K blocks
    (256, 1280, 2560, "swiglu"),       # exactly one token tile, few output tiles
    (257, 2560, 128, "shared_scale"),  # a second token tile of one token, K too short to share
    (700, 640, 1152, "store_bf16"),    # three token tiles, nine K blocks over a cluster
    (40, 19008, 128, "store_bf16"),    # more 128-row tiles than multiprocessors
    (1, 512, 640, "store_f32"),        # decode width: four row tiles, five K blocks shared in a cluster
    (16, 448, 1152, "gr_write"),       # decode width: a ragged fourth row tile, nine K blocks
])
def test_linear_fp8_small_and_middle_widths(T, n, k, kind, path):
    """The kernels of small and middle widths at the edges of their tiles and K shares, both routes, every epilogue."""
    torch = _torch()
    from fngine_b200 import linear
    weight = make_weight(torch, 7000 + T, n, k, T % 2 == 0)
    x = bf16_tensor(torch, synth.activations(70 + T, T, hidden=k))
    a = x.double()
    if path == "a8":
        xq, xs = linear.fp8_quantize_tokens(x)
        a = torch.from_numpy(O.e4m3_table().astype(np.float64)).cuda()[xq.long()] * xs.double()[:, None]
    make, ref, bf16_out = epilogue_case(torch, kind, T, n, exact_acc(torch, a, weight))
    work = linear.linear_fp8_workspace(weight, T)
    route = linear.L.FP8_PATH_A8 if path == "a8" else linear.L.FP8_PATH_AUTO
    epis = [make(), make()]
    for epi in epis:
        linear.linear_fp8(x, weight, epi, work, path=route)
    torch.cuda.synchronize()
    out, again = (e._keep[0] for e in epis)
    compare(torch, out, ref, bf16_out)
    assert torch.equal(out.view(torch.uint8), again.view(torch.uint8))  # repeated calls are bitwise identical


@pytest.mark.parametrize("T,n,k", [(1, 640, 512),       # decode width, few row tiles
                                   (16, 19072, 128),    # decode width, more row tiles than multiprocessors
                                   (17, 256, 256),      # middle widths
                                   (1100, 2560, 256)])  # the GEMM of two-SM tiles
def test_the_status_word_of_a_call_is_its_own(T, n, k):
    """Workspaces are not initialised by the caller: the status word, where an expired wait is recorded, reads 0 after a
    call on one full of ones."""
    torch = _torch()
    from fngine_b200 import linear
    weight = make_weight(torch, 5, n, k, False)
    x = bf16_tensor(torch, synth.activations(6, T, hidden=k))
    work = linear.linear_fp8_workspace(weight, T)
    work.fill_(255)
    out = torch.empty(T, n, dtype=torch.float32, device="cuda")
    linear.linear_fp8(x, weight, linear.store_f32(out), work)
    torch.cuda.synchronize()
    up = lambda v: (v + 255) // 256 * 256
    at = up(48 * k) + 256 if T <= 16 else up(2 * T * k) + up(4 * T)
    assert int(work[at:at + 4].view(torch.int32)) == 0
    compare(torch, out, exact_acc(torch, x.double(), weight), False)


@pytest.mark.parametrize("path", ["auto", "a8"])
@pytest.mark.parametrize("T,n,k,kind", [
    # two-SM tiles of 256 tokens x 256 rows, more of them than half of the GPU's pairs
    (1030, 5056, 384, "store_bf16"),    # ragged tokens and rows, three K blocks
    (1030, 5056, 384, "store_f32"),
    (769, 5056, 1152, "gr_write"),      # one token in the last tile
    (1025, 4736, 640, "shared_scale"),
    (1280, 4864, 256, "swiglu"),        # exact token tiles, a ragged last tile of 128 gate and 128 up rows
    (257, 19008, 128, "store_bf16"),    # the fewest tokens with a second tile, one K block
    # one-SM tiles: fewer tokens than such a tile takes, more than two waves of 128-row tiles
    (17, 38016, 128, "store_f32"),
    (130, 38080, 256, "store_bf16"),    # a second token tile of two tokens, a ragged last row tile
    (255, 38272, 128, "swiglu"),
    (129, 38080, 128, "shared_scale"),
    (40, 38080, 384, "gr_write"),
])
def test_linear_fp8_wide_tiles(T, n, k, kind, path):
    """The two GEMM kernels that middle widths do not take, at the edges of their tiles, both routes, every epilogue."""
    test_linear_fp8_small_and_middle_widths(T, n, k, kind, path)


@pytest.mark.parametrize("path", ["auto", "a8"])
@pytest.mark.parametrize("T,n,k,kind", [
    # (which units a count takes is asserted on the CPU, test_mid_units.py)
    (161, 1280, 2560, "swiglu"),        # units of 128 tokens: the first count that takes them, a ragged second unit
    (300, 2560, 6144, "gr_write"),      # three units, K over a cluster of two
    (193, 2560, 640, "shared_scale"),   # units of 128 in clusters of three: 64 would sum K in fewer chains
    (257, 2560, 640, "shared_scale"),   # units of 64 tokens, four chains for five K blocks, the last unit of one token
    (257, 2560, 896, "gr_write"),       # four chains of one, two, two and two K blocks
    (385, 1280, 896, "store_bf16"),     # units of 64 tokens in clusters of two, whose CTAs hold three and four chains
    (640, 2560, 640, "shared_scale"),   # the last count, too many units of 64 tokens for one wave: 128
    (512, 1408, 1280, "store_f32"),     # units of 128 would not fit beside each other: 256
    (255, 192, 128, "store_f32"),       # one K block, no cluster, half a row tile
    (999, 256, 2560, "store_bf16"),     # the activation kernel's last count with a block per token
    (1001, 256, 2560, "store_f32"),     # and its first with a warp per token, a ragged last block
    (1000, 384, 384, "store_bf16"),     # rows shorter than a warp's registers
])
def test_units_and_splits_chosen_by_the_token_count(T, n, k, kind, path):
    """The smaller units of the middle widths and the two forms of the activation kernel, at the counts where they change."""
    test_linear_fp8_small_and_middle_widths(T, n, k, kind, path)


@pytest.mark.parametrize("T,k", [(1001, 2560), (1004, 384), (1000, 2568)])
def test_token_pieces_of_many_tokens_are_bit_exact(T, k):
    """A warp per token (from 1000 tokens on, rows of at most 2560 values): codes, pieces and scales of whole and ragged blocks of
    eight tokens against the host's, with rows of zeros and tiny values. Longer rows take a block per token."""
    torch = _torch()
    from fngine_b200 import linear
    x = synth.activations(63, T, hidden=k) * np.logspace(-3, 3, T, dtype=np.float32)[:, None]
    x[5] = x[T - 1] = 0.0
    x[9, :100] *= 1e-4
    xb = synth.to_bf16_bits(x)
    xd = torch.from_numpy(xb.view(np.int16)).cuda().view(torch.bfloat16)
    codes, scales = linear.fp8_quantize_tokens(xd)
    want_c, want_s = O.quantize_tokens_e4m3(xb)
    assert np.array_equal(codes.cpu().numpy(), want_c)
    assert np.array_equal(scales.cpu().numpy().view(np.uint32), want_s.view(np.uint32))
    hi, lo, sc = linear.fp8_split_tokens(xd)
    w_hi, w_lo, w_sc = O.split_tokens_e4m3x2(xb)
    assert np.array_equal(hi.cpu().numpy(), w_hi) and np.array_equal(lo.cpu().numpy(), w_lo)
    assert np.array_equal(sc.cpu().numpy().view(np.uint32), w_sc.view(np.uint32))


def test_smaller_units_sum_in_shorter_chains():
    """300 tokens of 2560 x 6144 take units of 128 tokens in clusters of two, two chains of twelve K blocks in each CTA; the same
    rows among 641 tokens take units of 256 in clusters of two, one chain of 24. An fp32 chain's error grows with its length
    (0.82 of it measured here, 1 without the second chain), and it is the sums' only error: the inputs' products are exact."""
    torch = _torch()
    from fngine_b200 import linear
    n, k = 2560, 6144
    weight = make_weight(torch, 311, n, k, False)
    x = bf16_tensor(torch, synth.activations(312, 641, hidden=k))
    pieces = [p.cpu().numpy() for p in linear.fp8_split_tokens(x)]  # the values that the sums are of
    tab = O.e4m3_table().astype(np.float64)
    kept = torch.from_numpy((tab[pieces[0]] + tab[pieces[1]]) * pieces[2].astype(np.float64)[:, None]).cuda()
    ref = exact_acc(torch, kept[:300], weight)
    err = []
    for T in (300, 641):
        out = torch.full((T, n), float("nan"), dtype=torch.float32, device="cuda")
        linear.linear_fp8(x[:T], weight, linear.store_f32(out), linear.linear_fp8_workspace(weight, T))
        torch.cuda.synchronize()
        err.append(float((out[:300].double() - ref).norm() / ref.norm()))
    assert err[0] <= 0.9 * err[1] and err[1] <= 5e-6, err
