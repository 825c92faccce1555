// mvr_plan.hpp -- how a centroid-scoring call is laid out (host only; the kernels are
// in mvr_tc.cu).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace mvr {

constexpr int kPtTok = 128;            // tokens per MMA (M)
constexpr int kPtCtaTok = 2 * kPtTok;  // tokens per CTA = epilogue threads
constexpr int kPtCen = 128;            // centroids per tile (N): two source tiles

// Centroid scoring and top-nprobe per token (exact): how a call of n_tok tokens is
// laid out, and the sizes of its buffers in elements.
struct ProbePlan {
  uint32_t tiles_per_split, splits;  // 128-centroid tiles of a CTA, CTAs per token tile
  uint32_t k;                        // best scores kept: nprobe rounded up to a power of two
  uint32_t cap;                      // groups listed per token and split
  uint32_t list_at;                  // first flagged token in flags
  uint64_t cost;                     // waves x (centroid tiles of a CTA + 8)
  bool limited;                      // kProbeListBytes ruled out a cheaper split
  size_t n_ent, n_gid, n_cnt, n_flag, n_part;
};

// Most bytes of a launch's lists (36 a group, 4 a list); a handle keeps its largest.  One
// CTA per token tile fits at any nprobe (nprobe 32: 37,888 tokens, 0.74 GB).
constexpr size_t kProbeListBytes = 800u * 1000u * 1000u;

inline ProbePlan probe_plan(uint32_t n_tok, uint32_t n_cent, uint32_t nprobe, int n_sm) {
  ProbePlan p{};
  p.k = 1;
  while (p.k < nprobe) p.k *= 2;
  const uint32_t n_tiles = (n_cent + kPtCen - 1) / kPtCen;
  const uint32_t tok_tiles = std::max(1u, (n_tok + kPtCtaTok - 1) / kPtCtaTok);
  const uint32_t most = std::min(n_tiles, 2u * (uint32_t)n_sm / tok_tiles + 4u);
  // CTAs (one per SM at a time) per token tile: the count that takes the least
  // time, waves x (centroid tiles of a CTA + 8), 8 being what a split costs:
  // its start, and lists that fill from nothing
  // (a list's expected length is k (1 + ln(C / 8 k)) groups for scores in no
  // order, and a third more for those within 2 eps (unit vectors of 128
  // dimensions): 87 of 160 at k = 8 and 65,536 centroids, 14 of 48 at k = 1)
  uint32_t s = 1;
  uint64_t least = ~0ull;
  p.cost = ~0ull;
  auto cap_of = [&](uint32_t tiles) { return std::min(16u * p.k + 32u, tiles * (kPtCen / 8u)); };
  const bool any = (size_t)n_tok * most * (36u * cap_of(n_tiles) + 4u) <= kProbeListBytes;
  for (uint32_t c = 1; c <= most; c++) {
    const uint64_t waves = ((uint64_t)tok_tiles * c + n_sm - 1) / n_sm;
    const uint32_t tiles = (n_tiles + c - 1) / c;
    const uint64_t cost = waves * (tiles + 8u);
    least = std::min(least, cost);
    if (cost < p.cost && (any || c == 1 ||
                          (size_t)n_tok * ((n_tiles + tiles - 1) / tiles) *
                                  (36u * cap_of(tiles) + 4u) <= kProbeListBytes)) {
      p.cost = cost;
      s = c;
    }
  }
  p.limited = least < p.cost;
  p.tiles_per_split = (n_tiles + s - 1) / s;
  p.splits = (n_tiles + p.tiles_per_split - 1) / p.tiles_per_split;
  p.cap = cap_of(p.tiles_per_split);
  p.n_ent = (size_t)n_tok * p.splits * p.cap * 2;
  p.n_gid = (size_t)n_tok * p.splits * p.cap;
  p.n_cnt = (size_t)n_tok * p.splits;
  p.list_at = 2u + (n_tok + 63u) / 64u;
  p.n_flag = (size_t)p.list_at + n_tok;
  p.n_part = (size_t)n_sm * 64u * nprobe;
  return p;
}

// Tokens per launch: whole waves of token tiles, 4, 2 or 1 as the lists grow.  Where the
// lists' limit would leave such a launch fewer splits than it wants, launches of a half,
// third or quarter of that, if they cost less together (8 a launch): at 8,192 to 262,144
// centroids no more than 3 % above the unlimited plan's cost up to nprobe 16, 10 % at 32
// (whole launches alone: 32 and 70 %).  Measured at 65,536 centroids against the unlimited
// plan: 68,096 tokens x 8 probes 2.17 -> 1.84 ms and 2.0 -> 0.2 GB of lists, 31,488 x 32
// 3.56 -> 2.24 ms and 3.7 -> 0.7 GB.
inline uint32_t probe_chunk(uint64_t n_tok, uint32_t n_cent, uint32_t nprobe, int n_sm) {
  const uint32_t whole = (uint32_t)n_sm * kPtCtaTok * (nprobe == 1 ? 4u : nprobe <= 8 ? 2u : 1u);
  if (n_tok * 4u <= whole) return whole;  // nowhere near the limit, and a plan costs microseconds
  uint32_t chunk = whole;
  uint64_t least = ~0ull;
  for (uint32_t d = 1; d <= 4; d++) {
    const uint32_t t = (whole / d + kPtCtaTok - 1) / kPtCtaTok * kPtCtaTok;
    uint64_t cost = 0;
    bool limited = false;
    for (uint32_t n : {t, (uint32_t)(n_tok % t)}) {  // full launches, the last one
      const uint64_t times = n == t ? n_tok / t : n ? 1u : 0u;
      if (times == 0) continue;
      const ProbePlan p = probe_plan(n, n_cent, nprobe, n_sm);
      cost += (p.cost + 8u) * times;
      limited |= p.limited;
    }
    if (cost < least) { least = cost; chunk = t; }
    if (d == 1 && !limited) break;
  }
  return chunk;
}

// The same for tokens that arrive in n_part pieces (at most n_tok of them).
inline uint32_t score_chunk(uint32_t n_tok, uint32_t n_cent, uint32_t nprobe, int n_sm,
                            uint32_t n_part) {
  const uint32_t chunk = probe_chunk(n_tok, n_cent, nprobe, n_sm);
  return n_part > 1 ? std::min(chunk, ((n_tok / n_part + 255u) & ~255u)) : chunk;
}

}  // namespace mvr
