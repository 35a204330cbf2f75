"""The serial stretches of a decode layer on the GPU: the selection's short cuts, the fused layer of few tokens against the
separate calls, the host entry point's copies."""
import numpy as np
import pytest

from fngine_b200 import lib as L
from fngine_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu
H = 2560
IQ3_S, IQ4_NL, IQ2_S, IQ4_XS, Q2_0 = L.FMT_IQ3_S, L.FMT_IQ4_NL, L.FMT_IQ2_S, L.FMT_IQ4_XS, L.FMT_Q2_0


def _torch():
    import torch
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    return torch


def _bits(t):
    return t.contiguous().view(-1).cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("fg,fd,inter,tokens", [(IQ3_S, IQ3_S, 512, t) for t in (1, 2, 3, 4)] +
                         [(IQ3_S, IQ4_NL, 640, t) for t in (1, 2)] + [(IQ2_S, Q2_0, 640, t) for t in (1, 3)] +
                         [(IQ4_NL, IQ4_NL, 512, t) for t in (1, 3, 4, 11, 16)] + [(IQ4_XS, IQ4_NL, 640, t) for t in (1, 2)] +
                         [(IQ4_NL, Q2_0, 512, 7)])
def test_fused_layer_equals_the_four_calls(fg, fd, inter, tokens):
    """Both sides of the lines up to which values are their own arrival flags. Several calls on one workspace with other
    activations, so that a value of the call before would show; in one of them most tokens are alike (experts with many
    tokens, several passes; the pair visited last is not the one in the last slot)."""
    torch = _torch()
    from fngine_b200 import moe
    layer = moe.synth_layer(fg, fd, inter, 512, 40 + inter)
    ws, ws4 = moe.DecodeWorkspace(layer), moe.DecodeWorkspace(layer)
    wr = torch.from_numpy(synth.router_weights(303, rows=512).view(np.int16)).cuda().view(torch.bfloat16)
    y, y4 = (torch.empty(tokens, H, dtype=torch.float32, device="cuda") for _ in range(2))
    for call in range(5):
        x = torch.from_numpy(synth.activations(70 + call, tokens)).cuda()
        if call == 2:
            x[:tokens - tokens // 4] = x[0].clone()
        if call == 3:
            x = x.to(torch.bfloat16)
        y.fill_(float("nan"))
        moe.moe_layer_decode(wr, layer, x, ws, y)
        moe.moe_select_publish(ws.logits, x, None, 0, None, None, tokens, ws4)
        moe.moe_hot_gate_up(layer, tokens, ws4)
        moe.moe_hot_down(layer, tokens, ws4)
        moe.moe_combine(ws4, None, None, 0, None, None, None, y4, tokens)
        torch.cuda.synchronize()
        assert ws.status() == 0 and ws4.status() == 0
        assert np.array_equal(_bits(y), _bits(y4)), call
        n = 10 * tokens
        assert np.array_equal(ws.h(n).view(np.uint32), ws4.h(n).view(np.uint32))
        assert np.array_equal(ws.partial(n).view(np.uint32), ws4.partial(n).view(np.uint32))
        a, b = ws.work(), ws4.work()
        assert (a.n_items, a.n_pairs) == (b.n_items, b.n_pairs)
        for t in range(tokens):
            assert list(a.token_pairs[t]) == list(b.token_pairs[t]) and list(a.topk_weight[t]) == list(b.topk_weight[t])


@pytest.mark.parametrize("tokens", [4, 5])
def test_fused_layer_equals_the_four_calls_with_q2_0_down(tokens):
    """The two sides of the line of IQ4_NL + Q2_0 at 512."""
    test_fused_layer_equals_the_four_calls(IQ4_NL, Q2_0, 512, tokens)


@pytest.mark.parametrize("fg,fd,inter,tokens", [(IQ3_S, IQ3_S, 512, 1), (IQ3_S, IQ3_S, 512, 4), (IQ4_NL, IQ4_NL, 512, 16),
                                                (IQ2_S, Q2_0, 640, 1), (IQ3_S, IQ4_NL, 640, 2)])
def test_down_alone_behind_the_fused_layer(fg, fd, inter, tokens):
    """Both forms of the hand-off leave h re-quantized in the workspace: the down projection, run again by itself, gives the
    partial rows once more."""
    torch = _torch()
    from fngine_b200 import moe
    layer = moe.synth_layer(fg, fd, inter, 512, 60 + inter)
    ws = moe.DecodeWorkspace(layer)
    wr = torch.from_numpy(synth.router_weights(303, rows=512).view(np.int16)).cuda().view(torch.bfloat16)
    x = torch.from_numpy(synth.activations(77, tokens)).cuda()
    y, y2 = (torch.empty(tokens, H, dtype=torch.float32, device="cuda") for _ in range(2))
    moe.moe_layer_decode(wr, layer, x, ws, y)
    ws._view(ws.ws.partial, 10 * tokens * H * 4).fill_(255)
    moe.moe_hot_down(layer, tokens, ws)
    moe.moe_combine(ws, None, None, 0, None, None, None, y2, tokens)
    torch.cuda.synchronize()
    assert ws.status() == 0 and torch.equal(y, y2)


def test_values_that_are_not_numbers_arrive_too():
    """Rows of h that are NaN or infinite (an activation at the top of the range) must not be taken for missing ones."""
    torch = _torch()
    from fngine_b200 import moe
    layer = moe.synth_layer(IQ3_S, IQ3_S, 512, 512, 4)
    ws = moe.DecodeWorkspace(layer)
    wr = torch.from_numpy(synth.router_weights(303, rows=512).view(np.int16)).cuda().view(torch.bfloat16)
    x = torch.from_numpy(synth.activations(3, 2)).cuda()
    x[1] *= 1e36
    y = torch.empty(2, H, dtype=torch.float32, device="cuda")
    moe.moe_layer_decode(wr, layer, x, ws, y)
    torch.cuda.synchronize()
    assert ws.status() == 0
    assert torch.isfinite(y[0]).all() and not torch.isfinite(y[1]).all()


def _edge_logits(tokens):
    rng = np.random.default_rng(8)
    lg = rng.standard_normal((tokens, 512)).astype(np.float32)
    special = []
    special.append(np.full(512, 0.25, np.float32))                    # all equal: more than 32 survivors
    a = np.full(512, -np.inf, np.float32); a[[3, 77, 500]] = [1, 2, 3]; special.append(a)  # the bound is -infinity
    a = np.full(512, np.nan, np.float32); a[5:17] = np.arange(12); special.append(a)       # NaN never wins
    a = np.zeros(512, np.float32); a[::2] = -0.0; a[:6] = [5, 4, 3, 2, 1, 0.5]; special.append(a)  # -0 equals +0
    a = lg[0].copy(); a[40:72] = 9.0; special.append(a)               # exactly 32 survivors
    a = lg[0].copy(); a[40:73] = 9.0; special.append(a)               # 33
    a = lg[0].copy(); a[10:19] = np.inf; a[19] = np.nan; special.append(a)
    a = np.sort(lg[0]); special.append(a)                             # the largest logits in neighbouring lanes
    a = lg[0].copy(); a[[0, 32, 64, 96, 128, 160, 192, 224, 256, 288, 320]] = 7.0; special.append(a)  # all in one lane
    return lg, special


@pytest.mark.parametrize("tokens", [1, 3, 4, 16])
def test_selection_at_the_edges_of_its_pruning(tokens):
    torch = _torch()
    from fngine_b200 import moe
    layer = moe.synth_layer(IQ3_S, IQ3_S, 512, 512, 4)
    ws = moe.DecodeWorkspace(layer)
    lg, special = _edge_logits(tokens)
    x = torch.from_numpy(synth.activations(3, tokens)).cuda()
    for first in range(0, len(special), tokens):
        rows = lg.copy()
        for t, s in enumerate(special[first:first + tokens]):
            rows[t] = s
        full = np.zeros((tokens, 513), np.float32)
        full[:, :512] = rows
        moe.moe_select_publish(torch.from_numpy(full).cuda(), x, None, 0, None, None, tokens, ws)
        torch.cuda.synchronize()
        ids, w = O.topk(rows)
        work = ws.work()
        for t in range(tokens):
            assert list(work.topk_expert[t]) == list(ids[t]), (first, t)
            got = np.array(work.topk_weight[t], np.float32)
            assert np.array_equal(np.isnan(got), np.isnan(w[t]))
            assert np.nanmax(np.abs(got - w[t]), initial=0.0) <= 1e-6  # expf, a few ulp


@pytest.mark.parametrize("kind", ["pageable", "unaligned"])
@pytest.mark.parametrize("bf16", [False, True])
def test_host_activations_that_take_the_copy(kind, bf16):
    torch = _torch()
    from fngine_b200 import moe
    tokens = 3
    layer = moe.synth_layer(IQ3_S, IQ3_S, 512, 512, 9)
    ws = moe.DecodeWorkspace(layer)
    wr = torch.from_numpy(synth.router_weights(303, rows=512).view(np.int16)).cuda().view(torch.bfloat16)
    x = torch.from_numpy(synth.activations(12, tokens)).to(torch.bfloat16 if bf16 else torch.float32)
    if kind == "unaligned":
        flat = torch.empty(tokens * H + 1, dtype=x.dtype).pin_memory()
        xh = flat[1:].view(tokens, H)
        xh.copy_(x)
    else:
        xh = x
    xd = torch.empty(tokens, H, dtype=x.dtype, device="cuda")
    yd, y2 = (torch.empty(tokens, H, dtype=torch.float32, device="cuda") for _ in range(2))
    yh = torch.empty(tokens, H, dtype=torch.float32).pin_memory()
    pinned = x.clone().pin_memory()
    for src in (xh, pinned):
        yh.zero_()
        xd.zero_()
        moe.moe_layer_decode_host(wr, layer, src, ws, xd, yd, yh)
        moe.moe_layer_decode(wr, layer, x.cuda(), ws, y2)
        torch.cuda.synchronize()
        assert np.array_equal(yh.numpy().view(np.uint32), y2.cpu().numpy().view(np.uint32))
        assert torch.equal(xd.cpu(), x)


def test_host_buffers_over_two_registrations():
    """x and y that each lie in two neighbouring page-locked ranges: read and written in place, the same bits."""
    torch = _torch()
    import mmap
    from fngine_b200 import moe
    tokens = 2
    layer = moe.synth_layer(IQ3_S, IQ3_S, 512, 512, 9)
    ws = moe.DecodeWorkspace(layer)
    wr = torch.from_numpy(synth.router_weights(303, rows=512).view(np.int16)).cuda().view(torch.bfloat16)
    x = torch.from_numpy(synth.activations(13, tokens))
    mem = torch.frombuffer(mmap.mmap(-1, 16 * 4096), dtype=torch.float32)  # x and y: five pages each
    xh, yh = mem[:tokens * H].view(tokens, H), mem[5 * 1024:5 * 1024 + tokens * H].view(tokens, H)
    xh.copy_(x)
    cudart, base, pages = torch.cuda.cudart(), mem.data_ptr(), [0, 2, 7, 10]
    for a, b in zip(pages, pages[1:]):
        assert int(cudart.cudaHostRegister(base + 4096 * a, 4096 * (b - a), 0)) == 0
    try:
        xd = torch.zeros(tokens, H, dtype=torch.float32, device="cuda")
        yd, y2 = (torch.empty(tokens, H, dtype=torch.float32, device="cuda") for _ in range(2))
        yd.fill_(7.0)
        moe.moe_layer_decode_host(wr, layer, xh, ws, xd, yd, yh)
        moe.moe_layer_decode(wr, layer, x.cuda(), ws, y2)
        torch.cuda.synchronize()
        assert np.array_equal(yh.numpy().view(np.uint32), y2.cpu().numpy().view(np.uint32))
        assert torch.equal(xd.cpu(), x) and bool((yd == 7.0).all())  # (the result went past the device buffer)
    finally:
        torch.cuda.synchronize()
        for a in pages[:-1]:
            cudart.cudaHostUnregister(base + 4096 * a)


def test_page_locked_buffers_on_a_thread_without_a_context():
    torch = _torch()
    import ctypes as C
    import threading
    from fngine_b200 import moe
    tokens = 1
    layer = moe.synth_layer(IQ3_S, IQ3_S, 512, 512, 9)
    ws = moe.DecodeWorkspace(layer)
    wr = torch.from_numpy(synth.router_weights(303, rows=512).view(np.int16)).cuda().view(torch.bfloat16)
    xh = torch.from_numpy(synth.activations(14, tokens)).pin_memory()
    xd = torch.zeros(tokens, H, dtype=torch.float32, device="cuda")
    yd, y2 = (torch.full((tokens, H), 7.0, dtype=torch.float32, device="cuda") for _ in range(2))
    yh = torch.empty(tokens, H, dtype=torch.float32).pin_memory()
    torch.cuda.synchronize()
    status = []

    def call():
        status.append(L.load().fb_moe_layer_decode_host(wr.data_ptr(), C.byref(layer.layout), xh.data_ptr(), L.DT_F32, tokens,
                                                        C.byref(ws.ws), ws.logits.data_ptr(), xd.data_ptr(), yd.data_ptr(),
                                                        yh.data_ptr(), None))
    t = threading.Thread(target=call)
    t.start()
    t.join()
    moe.moe_layer_decode(wr, layer, xh.cuda(), ws, y2)
    torch.cuda.synchronize()
    assert status == [0] and bool((yd == 7.0).all())
    assert np.array_equal(yh.numpy().view(np.uint32), y2.cpu().numpy().view(np.uint32))


@pytest.mark.parametrize("fg,fd,inter", [(IQ3_S, IQ3_S, 512), (IQ4_NL, IQ4_NL, 512), (IQ3_S, IQ4_NL, 640)])
@pytest.mark.parametrize("fused", [True, False])
def test_a_value_that_does_not_arrive_in_time(fg, fd, inter, fused):
    """One poll for what other multiprocessors write instead of millions, at one token, where h is never there when the first
    down tile wants it: rows that are their own arrival flags (the fused layer) and an item's flag (behind a stand-alone
    selection). The layer ends by itself in a few seconds, the status says why, and the next layer on the workspace gives the
    right bits."""
    torch = _torch()
    import time
    from fngine_b200 import moe
    layer = moe.synth_layer(fg, fd, inter, 512, 21)
    ws = moe.DecodeWorkspace(layer)
    wr = torch.from_numpy(synth.router_weights(303, rows=512).view(np.int16)).cuda().view(torch.bfloat16)
    x = torch.from_numpy(synth.activations(15, 1)).cuda()
    want, y = (torch.empty(1, H, dtype=torch.float32, device="cuda") for _ in range(2))

    def run(out):
        if fused:
            moe.moe_layer_decode(wr, layer, x, ws, out)
        else:
            moe.moe_select_publish(ws.logits, x, None, 0, None, None, 1, ws)
            moe.moe_hot_experts(layer, 1, ws)
            moe.moe_combine(ws, None, None, 0, None, None, None, out, 1)
        torch.cuda.synchronize()

    moe.moe_layer_decode(wr, layer, x, ws, want)
    run(y)
    assert ws.status() == 0 and torch.equal(y, want)
    ws.ws.wait_polls = 1
    began = time.monotonic()
    run(y)
    assert time.monotonic() - began < 10.0
    assert ws.status() == L.STATUS_PIPELINE_TIMEOUT
    ws.ws.wait_polls = 0
    ws._view(ws.ws.status, 4).zero_()
    y.fill_(float("nan"))
    run(y)
    assert ws.status() == 0 and torch.equal(y, want)
