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


def _function(name):
    text = _source()
    at = text.index("{", text.index(name + "(const RingN<S>& r"))
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i]


def test_an_expired_wait_is_not_overwritten_by_the_producers_count():
    """Every warp learns of an expired wait from the end mark. It is written when the ring is made, by an abort, and by the
    producer in the place of the first value only."""
    text = _source()
    assert sorted(re.findall(r"end_seq\s*=[^=][^;]*;", text)) == ["end_seq = 0;", "end_seq = kRingOpen;"]
    assert "*r.end_seq = 0;" in _function("void ring_abort")
    assert "atomicCAS(const_cast<int*>(r.end_seq), kRingOpen, entries)" in _function("void ring_close")
    assert len(re.findall(r"atomic\w+\([^;]*end_seq", text)) == 1


def test_a_block_waits_for_its_copies_behind_an_expired_wait():
    """Whoever gives up waits (bounded) until the producer has stopped and the last staged entries' copies have landed; the
    producer does so when it has stopped for another warp's sake too. Those barriers want an arrival of every quantizing warp,
    so these go on to the last staged entry."""
    text = _source()
    assert "mbar_wait_hint(&r.full[e % S]" in _function("void ring_drain")
    for m in re.finditer(r"ring_abort\(r(?:ing)?, \w+(?:\.status)?\);", text):  # consumers: at once
        behind = text[m.end():m.end() + 120]
        where = text[:m.start()]
        if where.rfind("draw_task_n(") > where.rfind("experts_kernel(") or where.rfind("combine_tile_direct(") > where.rfind("experts_kernel("):
            assert "ring_drain(" in behind
    body = _kernel()
    start = body.index("if (warp == C::kWarps)")
    producer = body[start:body.index("if (DIRECT && warp > C::kWarps)")]
    mark = producer[producer.index("~EndMark()"):]
    assert mark.index("ring_close(r, i);") < mark.index("if (failed) ring_drain(r);")
    seen = producer[producer.index("*ring.end_seq == 0"):]
    assert seen.index("failed = true;") < seen.index("return false;") < seen.index("mbar_wait_hint(&ring.empty[s]")
    # the producer may sit in its wait for a slot (2^21 tries of a microsecond): those who need it to stop wait longer
    assert re.search(r"kStopPolls = 1u << 26;", _source()) and "i < kStopPolls" in _function("void ring_drain")
    assert "++tries > kStopPolls" in _quantizers()
    text = _quantizers()
    assert "*ring.staged_seq, 0)) <= uint32_t(seq)" in text and "end_seq, 0) <= seq" not in text
    assert text.count("return;") == 2 and text.index("if (expired && lane == 0) ring_drain(ring);") < text.rindex("return;")
