"""How the middle-width FP8 projection is cut into units (csrc/mid_units.h), compiled with the host compiler: the tokens of a unit
and the CTAs that share its K, for a B200's multiprocessors and clusters. No GPU."""
import itertools
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "fngine_b200", "csrc")
SMS, RESIDENT = 148, [0, 148, 74, 45, 33, 26, 22, 15, 15]  # clusters of 0..8 CTAs at once, as the driver counts them
PROGRAM = r"""
#include "mid_units.h"
#include <cstdio>
#include <cstdlib>
// multiprocessors, resident clusters of 0..8 CTAs; then from the input: tokens, row tiles, K blocks, pieces of every question
int main(int, char** argv) {
  int resident[9], t, m, kb, p;
  for (int i = 0; i < 9; ++i) resident[i] = atoi(argv[2 + i]);
  while (scanf("%d %d %d %d", &t, &m, &kb, &p) == 4) {
    const fb::MidUnits a = fb::mid_units(t, m, kb, p, atoi(argv[1]), resident);
    const fb::MidUnits b = fb::mid_units_of(fb::kMidTok, t, m, kb, resident);
    printf("%d %d %d %d %d %d %d %d\n", a.tile, a.cluster, a.chains, a.slots, a.units, b.cluster, b.chains, b.units);
  }
}
"""


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    d = tmp_path_factory.mktemp("mid_units")
    (d / "p.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", CSRC, str(d / "p.cpp"), "-o", str(d / "p")])
    args = [str(d / "p"), str(SMS)] + [str(r) for r in RESIDENT]

    def run(questions):
        text = "\n".join(" ".join(str(v) for v in q) for q in questions)
        out = subprocess.run(args, input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(int(v) for v in line.split()) for line in out.splitlines()]
    return run


def longest_chain(kb, cluster, per_cta):
    """K blocks of the longest chain, by the kernel's own division: K over the cluster's CTAs, a CTA's part over its chains."""
    longest = 0
    for rank in range(cluster):
        own = kb * (rank + 1) // cluster - kb * rank // cluster
        n = min(own, per_cta)
        longest = max([longest] + [own * (c + 1) // n - own * c // n for c in range(n)])
    return longest


@pytest.mark.parametrize("tokens,m_tiles,kb,pieces,tile,cluster", [
    # the cases of the GPU test of the counts where units change, and what each of them is for
    (161, 10, 20, 2, 128, 6),   # 1280 x 2560 SwiGlu: the first count, a ragged second unit
    (300, 20, 48, 2, 128, 2),   # 2560 x 6144: three units, K over a cluster of two
    (193, 20, 5, 2, 128, 3),    # 2560 x 640: units of 64 would sum K in fewer chains
    (257, 20, 5, 2, 64, 1),     # 2560 x 640: units of 64, four chains for five K blocks, a last unit of one token
    (257, 20, 5, 1, 64, 1),
    (640, 20, 5, 2, 128, 1),    # the last count, too many units of 64 for one wave
    (257, 20, 7, 2, 64, 1),     # 2560 x 896: four chains of one, two, two and two K blocks
    (385, 10, 7, 2, 64, 2),     # 1280 x 896: units of 64 in clusters, CTAs of three and of four chains, a last unit of one token
    (385, 10, 7, 1, 64, 2),
    (255, 2, 1, 2, 64, 1),      # 192 x 128: one K block
    # outside of the range, and where smaller units would cost more than they give
    (160, 20, 5, 2, 256, 5), (641, 20, 5, 2, 256, 2),
    (512, 11, 10, 2, 256, 6),   # 44 of 45 clusters of three
    (256, 13, 10, 2, 256, 8),   # 26 of 26 clusters of five
    (512, 10, 10, 2, 128, 3),   # 40 of 45
    (384, 11, 21, 2, 128, 4),   # 33 of 33 clusters of four
    (600, 5, 21, 2, 128, 5),    # 25 of 26 clusters of five
    (170, 32, 10, 2, 256, 4),   # half as much again taken in, for two tiles of 128 and 42 tokens
    (193, 32, 10, 2, 128, 2),
    (170, 48, 4, 2, 64, 1),     # 6144 x 512
])
def test_units_of_known_calls(ask, tokens, m_tiles, kb, pieces, tile, cluster):
    assert ask([(tokens, m_tiles, kb, pieces)])[0][:2] == (tile, cluster)


def test_smaller_units_keep_the_chains_one_wave_and_room(ask):
    """For every shape: K in no fewer chains than units of 256 have and none longer than theirs, all CTAs in one wave, an eighth
    of the multiprocessors free beside clusters of an odd size, tiles that cover the tokens."""
    questions = list(itertools.product(list(range(1, 660, 13)) + [160, 161, 192, 193, 256, 257, 640, 641],
                                       range(1, 80, 3), list(range(1, 13)) + [16, 20, 21, 24, 32, 48], (1, 2)))
    smaller = 0
    for (tokens, m, kb, _), (tile, cluster, chains, slots, units, c256, chains256, _) in zip(questions, ask(questions)):
        assert tile in (64, 128, 256) and units == m * -(-tokens // tile) and 1 <= cluster <= min(kb, 8)
        assert slots % 32 == 0 and min(tokens, tile) <= slots <= tile
        if tile == 256:
            assert cluster == c256
            continue
        smaller += 1
        assert 160 < tokens <= 640 and units <= RESIDENT[cluster] and units * cluster <= SMS
        assert chains >= chains256 and longest_chain(kb, cluster, 256 // tile) <= longest_chain(kb, c256, 1)
        assert cluster == 1 or cluster % 2 == 0 or 8 * units * cluster <= 7 * SMS
    assert smaller > 1000
