"""Rules that the expert kernel's ring keeps in its source (csrc/moe_decode_experts.cuh): a race or a copy in flight at a
block's end shows on a GPU by chance only. No GPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "fngine_b200", "csrc")


def _source():
    with open(os.path.join(CSRC, "moe_decode_experts.cuh")) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _kernel():
    text = _source()
    return text[text.index("experts_kernel(fb_moe_expert_layout L"):]


def _quantizers():
    body = _kernel()
    start = body.index("if (DIRECT && warp > C::kWarps)")
    return body[start:body.index("const uint32_t sign_base", start)]


def test_a_quantizing_warp_reads_an_entry_behind_its_barrier():
    """Only an acquire orders the warp's writes into the slot behind the consumers' reads of the entry before, and its reads of
    the description behind the producer's stores."""
    text = _quantizers()
    wait = text.index("mbar_test_wait(&ring.staged[s]")
    reads = [m.start() for m in re.finditer(r"ring\.meta|s_meta|ld\.volatile", text)]
    assert reads and min(reads) > wait and "ld.volatile" not in text


def test_the_barrier_follows_the_description_and_every_entry_waits_for_the_quantizing_warps():
    body = _kernel()
    store, staged = body.index("m->store("), body.index("mbar_arrive(&ring.staged[s])")
    assert store < staged < body.index("mbar_arrive(full)", staged)
    text = _quantizers()  # gate/up entries too: the producer cannot lap a warp, so an entry's phase is its own
    gate_up = text[text.index("if (kind == 0)"):]
    assert gate_up.index("mbar_arrive(&ring.full[s])") < gate_up.index("continue")
    assert "mbar_arrive_n" not in body
