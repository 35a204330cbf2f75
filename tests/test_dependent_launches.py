"""Rules that the CUDA sources keep where launches are chained by programmatic dependent launch. A kernel launched that way
may start while its predecessor runs, so what keeps its reads in order is in the source and can be checked there (a
race on the GPU shows by chance only). The same for what a kernel does once a bounded wait has run out. No GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "fngine_b200", "csrc")
KERNEL = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)\s*)?(\w+)\s*\(")


def _block(text, at, opening, closing):
    """The text from the bracket at `at` to its match, and the position behind it."""
    depth = 0
    for i in range(at, len(text)):
        if text[i] == opening:
            depth += 1
        elif text[i] == closing:
            depth -= 1
            if depth == 0:
                return text[at:i + 1], i + 1
    raise AssertionError("unbalanced source")


def kernels():
    """name -> (parameters, body) of every kernel, comments removed."""
    found = {}
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
        for m in KERNEL.finditer(text):
            params, end = _block(text, m.end() - 1, "(", ")")
            body, _ = _block(text, text.index("{", end), "{", "}")
            found[m.group(1)] = (params, body)
    return found


KERNELS = kernels()
CHAINED = sorted(n for n, (_, body) in KERNELS.items() if "pdl_wait_prior()" in body)


def test_the_sources_are_read():
    assert len(KERNELS) > 25 and {"experts_kernel", "grouped_kernel", "fp8_mid_kernel", "pf_combine_kernel"} <= set(CHAINED)


@pytest.mark.parametrize("split", ["fp8_split_tokens_kernel", "fp8_quantize_tokens_kernel"])
def test_a_split_waits_before_it_lets_the_projection_start(split):
    """fp8_decode_kernel and fp8_mid_kernel ask for weight codes before their own wait. That is in order only if everything
    ahead of the activation split, which may have written the codes, is complete when the split lets them start."""
    body = KERNELS[split][1]
    assert body.count("pdl_wait_prior()") == 1 and body.count("pdl_launch_dependents()") == 1
    assert body.index("pdl_wait_prior()") < body.index("pdl_launch_dependents()")


@pytest.mark.parametrize("name", CHAINED)
def test_no_load_of_a_chained_kernel_may_move_ahead_of_its_wait(name):
    """Loads through const __restrict__ parameters and by __ldg count as invariant: the compiler may move them ahead of the
    wait, where the predecessor's data is not there yet."""
    params, body = KERNELS[name]
    assert "__restrict__" not in params and "__ldg(" not in body


def test_no_helper_of_the_chained_kernels_uses_invariant_loads():
    for name in sorted(os.listdir(CSRC)):
        if name == "probes.cu":  # (ordinary launches)
            continue
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
        assert "__ldg(" not in text, name
        for m in re.finditer(r"__device__ __forceinline__[^;{]*\([^{;]*\{", text):
            assert "__restrict__" not in m.group(0), (name, m.group(0)[:80])


@pytest.mark.parametrize("name", ["fp8_small_kernel", "fp8_mid_kernel"])
def test_a_cluster_with_a_missing_partial_tile_stores_nothing(name):
    """Every CTA learns of an expired wait anywhere in its cluster at the barrier that ends the sums, and the outputs
    stand behind that."""
    body = KERNELS[name][1]
    tell, learn = body.find("st_cluster_u32(&bars->failed"), body.find("bool complete")
    assert 0 <= tell < learn
    barrier = body.rindex("cluster_sync()", 0, learn)
    guard = re.search(r"(for|if) \([^{]*\bcomplete &&[^{]*\{", body)
    assert tell < barrier and learn < guard.start()
    _, end = _block(body, guard.end() - 1, "{", "}")
    stores = [m.start() for m in re.finditer(r"static_cast<(?:__nv_bfloat16|float)\*>\(a\.out\)", body) if m.start() > barrier]
    assert stores and all(guard.start() < at < end for at in stores)


def test_lanes_read_behind_the_acquire_of_lane_0():
    """A shuffle orders no memory: between lane 0's acquiring atomic and the other lanes' loads stands a __syncwarp."""
    with open(os.path.join(CSRC, "moe_decode.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    body, _ = _block(text, text.index("{", text.index("void item_contribution_done")), "{", "}")
    behind = body[body.index("atom.acq_rel"):body.index("quantize_h_row")]
    assert "__syncwarp();" in behind
