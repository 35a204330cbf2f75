"""Which host buffers a kernel may read and write in place: the walk over page-locked ranges (csrc/host_range.h), compiled with
the host compiler and asked about made-up registrations. No GPU."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "fngine_b200", "csrc")
PROGRAM = r"""
#include "host_range.h"
#include <cstdio>
#include <cstdlib>
// host bytes, then start, size, device address of every registration -> device address or 0, and the questions asked
int main(int argc, char** argv) {
  auto n = [&](int i) { return uintptr_t(strtoull(argv[i], nullptr, 0)); };
  int asked = 0;
  const uintptr_t r = fb::pinned_range(n(1), size_t(n(2)), [&](uintptr_t p, fb::PinnedByte& b) {
    ++asked;
    for (int i = 3; i + 2 < argc; i += 3)
      if (p >= n(i) && p - n(i) < n(i + 1)) {
        b = {n(i + 2) + (p - n(i)), n(i), size_t(n(i + 1))};
        return true;
      }
    return false;
  });
  std::printf("%llu %d\n", (unsigned long long)r, asked);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("host_range")
    (d / "p.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-I", CSRC, str(d / "p.cpp"), "-o", str(d / "p")])
    return str(d / "p")


def ask(program, host, size, *ranges):
    flat = [str(v) for r in ranges for v in r]
    return tuple(int(v) for v in subprocess.check_output([program, str(host), str(size)] + flat).split())


P = 4096


@pytest.mark.parametrize("host,size,ranges,device,asked", [
    (P, P, [(P, P, 70 * P)], 70 * P, 1),                                      # the buffer is the registration
    (P + 48, 100, [(P, P, 70 * P)], 70 * P + 48, 1),                          # inside it
    (P, 1, [(P, P, 70 * P)], 70 * P, 1),
    (P + 48, P, [(P, P, 70 * P)], 0, 2),                                      # the registration ends inside the buffer
    (P, P + 1, [(P, P, 70 * P)], 0, 2),                                       # one byte short
    (2 * P - 1, 2, [(P, P, 70 * P)], 0, 2),                                   # only the first byte is held
    (P, P, [(P + 16, P, 70 * P)], 0, 1),                                      # it begins inside the buffer
    (P, 3 * P, [(P, P, 70 * P), (3 * P, P, 72 * P)], 0, 2),                   # both ends held, not the middle
    (P + 8, 2 * P - 16, [(P, P, 70 * P), (2 * P, P, 71 * P)], 70 * P + 8, 2),  # two neighbours, addresses in step
    (P, 2 * P, [(P, P, 70 * P), (2 * P, P, 90 * P)], 0, 2),                   # two neighbours mapped apart
    (P, P, [(P, P, 0)], 0, 1),                                                # no address on this device
    (P, P, [], 0, 1),                                                         # pageable
])
def test_a_buffer_is_page_locked_from_end_to_end_or_not_at_all(program, host, size, ranges, device, asked):
    assert ask(program, host, size, *ranges) == (device, asked)


def test_the_host_entry_asks_about_whole_buffers():
    with open(os.path.join(CSRC, "moe_decode.cu")) as f:
        text = f.read()
    body = text[text.index("int32_t fb_moe_layer_decode_host("):]
    assert "pinned_on_device(x_host, xb)" in body and "pinned_on_device(y_host, size_t(tokens) * H * 4)" in body
