// How fp8_mid_kernel's work is cut: tokens of a unit and CTAs of its cluster. Plain C++ without CUDA headers: the choice is
// tested with a host compiler.
#pragma once

namespace fb {

constexpr int kMidTok = 256, kMidMaxCluster = 8;
constexpr int kMidRowBytes = 128;                       // of a row of weights or activation codes in a K block
constexpr int kMidStageWeights = 128 * kMidRowBytes;    // 16 KB of weights a stage
// Bytes of a stage: the weights and `pieces` tiles of `tok` token slots.
constexpr int mid_stage(int pieces, int tok) { return kMidStageWeights + pieces * tok * kMidRowBytes; }

struct MidUnits {
  int tile;     // tokens of a unit: kMidTok or a power of two below it
  int cluster;  // CTAs that share a unit's K
  int chains;   // fp32 chains that a unit's K is summed in, over the cluster's CTAs and each one's tensor-memory columns
  int slots;    // token slots of a stage, a multiple of 32
  int units;    // row tiles x token tiles
};

// tokens x (m_tiles row tiles of 128 weight rows) x (kb K blocks of 128), activations in `pieces` codes; resident[c] = clusters of c
// CTAs that run at once, one CTA per multiprocessor; sms = multiprocessors.
inline MidUnits mid_units_of(int tile, int tokens, int m_tiles, int kb, const int* resident) {
  MidUnits u;
  u.tile = tile;
  u.units = m_tiles * ((tokens + tile - 1) / tile);
  u.cluster = kb < kMidMaxCluster ? kb : kMidMaxCluster;
  while (u.cluster > 1 && resident[u.cluster] < u.units) --u.cluster;
  const int chains = u.cluster * (kMidTok / tile);
  u.chains = chains < kb ? chains : kb;
  u.slots = ((tokens < tile ? tokens : tile) + 31) & ~31;
  return u;
}

// A unit has 256 tokens, but where a few hundred tokens make one wave of smaller units, 128, or 64 where K is short: the partial
// tile and the outputs are then shared out more evenly. Conditions, with both sides in us per call, units of 256 and smaller ones,
// in captured graphs of such calls on different weights (exact activations):
// - 161 to 640 tokens. Below, the intake that doubles costs more than the shares give: 2560 x 640 at 65 8.5 and 9.7, 1280 x 2560 GrWrite
//   at 130 12.9 and 14.3 (but 256 x 896 at 130 9.1 and 7.6). Above it is mixed, and not taken: 2560 x 640 at 700 33.9 and 28.2, 1280 x 2560
//   SwiGlu at 800 20.5 and 17.2, 192 x 4096 at 1600 19.1 and 23.2.
// - One wave, no fewer chains (the error against fp64 grows with a chain's length: 2560 x 6144 at 300 tokens 1.10e-6 in three,
//   1.27e-6 in two), and no more than 100 KB taken in by a CTA in addition. So: 1280 x 2560 SwiGlu at 200 12.2 and 11.5, at 300
//   15.5 and 12.4; 2560 x 640 at 300 22.4 and 17.2, at 640 32.9 and 28.1; 2560 x 6144 at 300 34.7 and 29.7.
// - Clusters of an odd size leave an eighth of the multiprocessors free. Behind the activation kernel, whose blocks end one by one, the
//   last of them find no room although `resident` has it, and the call takes two waves: 1408 x 1280 at 512 (44 of 45 clusters
//   of three) 14.6 and 19.2, 1152 x 1280 at 620 (45 of 45) 16.6 and 20.7, 1664 x 1280 at 256 (26 of 26 of five) 13.0 and 16.2. 42 of 45 and
//   24 of 26 are 12 to 20 % faster than units of 256; 25 of 26 is faster but where all its tiles are full (640 x 2688 at 600
//   15.1 and 14.6, at 640 15.2 and 16.1). Clusters of two, four and six run at their last place.
// - Up to 192 tokens, clusters of units of 128 take in at most a quarter more: 4096 x 1280 at 170 13.7 and 14.6, 1792 x 3072 at 161 11.9 and
//   13.1 (both half as much again); 1536 x 2560 at 192 (a fifth) 12.2 and 12.0. Single CTAs and units of 64 gain with any.
inline MidUnits mid_units(int tokens, int m_tiles, int kb, int pieces, int sms, const int* resident) {
  const MidUnits whole = mid_units_of(kMidTok, tokens, m_tiles, kb, resident);
  if (tokens <= 160 || tokens > 640) return whole;
  auto intake = [&](const MidUnits& u) { return kb * mid_stage(pieces, u.slots) / u.cluster; };  // bytes, of a CTA
  for (int tile = kb <= 8 ? 64 : 128; tile < kMidTok; tile *= 2) {
    const MidUnits u = mid_units_of(tile, tokens, m_tiles, kb, resident);
    if (u.units > sms || u.chains < whole.chains || intake(u) > intake(whole) + 100 * 1024) continue;
    if (u.cluster > 1 && u.cluster % 2 == 1 && 8 * u.units * u.cluster > 7 * sms) continue;
    if (tile == 128 && u.cluster > 1 && tokens <= 192 && 4 * intake(u) > 5 * intake(whole)) continue;
    return u;
  }
  return whole;
}

}  // namespace fb
