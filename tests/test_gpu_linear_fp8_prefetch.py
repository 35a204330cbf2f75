"""Decode-width FP8 projections that ask their weights into L2 ahead of the dependency wait: large matrices at the two sides
of the token limit, ragged last tiles, and weights that the kernel just before the call has written."""
import pytest

from fngine_b200 import synth
from test_gpu_linear_fp8_decode import _torch, bf16_tensor, compare, exact_acc, make_weight

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 4, 5])
@pytest.mark.parametrize("n,k,kind", [(9160, 2560, "store_f32"), (6544, 2560, "swiglu"), (3280, 2560, "store_bf16"), (3272, 2560, "store_f32")])
def test_weights_written_just_before_the_call(T, n, k, kind):
    torch = _torch()
    from fngine_b200 import linear
    sets = [make_weight(torch, 40 + i, n, k, False) for i in range(3)]
    weight = make_weight(torch, 60, n, k, False)
    work = linear.linear_fp8_decode_workspace(weight)
    x = bf16_tensor(torch, synth.activations(500 + T, T, hidden=k))
    outs = []
    for s in sets:  # back to back: call, new weights, call, new weights ...
        weight.codes.copy_(s.codes)
        weight.scales.copy_(s.scales)
        if kind == "swiglu":
            out = torch.full((T, n // 2), float("nan"), dtype=torch.bfloat16, device="cuda")
            linear.linear_fp8_decode(x, weight, linear.swiglu(out), work)
        else:
            out = torch.full((T, n), float("nan"), dtype=torch.bfloat16 if kind == "store_bf16" else torch.float32, device="cuda")
            linear.linear_fp8_decode(x, weight, getattr(linear, kind)(out), work)
        outs.append(out)
    torch.cuda.synchronize()
    for s, out in zip(sets, outs):
        acc = exact_acc(torch, x, s)
        g, u = acc[:, :n // 2], acc[:, n // 2:]
        compare(torch, out, g / (1.0 + torch.exp(-g)) * u if kind == "swiglu" else acc, kind != "store_f32")
