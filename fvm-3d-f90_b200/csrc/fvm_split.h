// fvm_split.h — how the z columns of a group's tiles become the tasks of its
// work queue. Host code without CUDA calls.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <cstddef>
#include <vector>

#include "fvm_types.h"

namespace fvm {

// Split nz planes into chunks of at most L planes, all of nearly equal length
// (lengths differ by at most one plane).
inline void equal_chunks(int64_t nz, int64_t L, std::vector<int64_t>& z0s) {
  z0s.clear();
  const int64_t nc = std::max<int64_t>(1, (nz + L - 1) / L);
  const int64_t base = nz / nc, extra = nz % nc;
  int64_t z = 0;
  for (int64_t c = 0; c < nc; ++c) {
    z0s.push_back(z);
    z += base + (c < extra ? 1 : 0);
  }
  z0s.push_back(nz);
}

// A z column of one tile.
struct ZColumn {
  int blk, x0, y0, nz;
};

// Cut the columns into equal chunks of at most L planes.
inline void chunk_columns(const std::vector<ZColumn>& cols, int64_t L, std::vector<Task>& out) {
  std::vector<int64_t> z0s;
  for (const auto& c : cols) {
    equal_chunks(c.nz, L, z0s);
    for (size_t i = 0; i + 1 < z0s.size(); ++i) out.push_back({c.blk, c.x0, c.y0, (int)z0s[i], (int)z0s[i + 1], 0});
  }
}

struct Split {
  double share;  // plane-times of a CTA
  int tries;     // shares tried
};

// Even split of z columns over `slots` resident CTAs: the columns, taken one
// after the other, are cut wherever a CTA's share of the work is full, so all
// shares are the same to within a plane or two. While the columns do not
// outnumber the slots a stage is one round of the queue (equal chunks leave
// CTAs idle in its last round: 2.3 rounds on the 128^3 vortex, 0.8 of one on a
// 61x83x47 blast); more columns stay whole but for the few where a share ends,
// and the queue, longest first, evens them out. A piece of c planes costs
// c + ovh plane-times (the z window's warm-up and the set-up) and has at least
// kMinPiece planes where the column allows it. The smallest share that fits is
// found by growing it from what fits at least, O(pieces) per try: the mean of
// the planes plus one piece's ovh, or the mean of the columns with an ovh each
// if that is more (columns of a plane or two). One to eight tries in the tests (4,000 blocks
// of 33x17x2 from the first bound alone: 36), so the re-plans of a serving
// loop stay cheap. Measured per step, equal chunks of
// the length a queue estimate picked -> even split: vortex 128^3 FP64 926 ->
// 909 us, 64^3 172 -> 153; Taylor-Green 128^3 FP64 877 -> 833, 30^3 FP32 96 ->
// 74; 61x83x47 blast FP64 159 -> 138; 24 mixed FP32 cases 1143 -> 1086. The
// pieces' least length (1 to 3) and ovh (0.6 to 1.4 for WENO) move these by
// less than 2 %.
inline Split even_split(const std::vector<ZColumn>& cols, int slots, double ovh, std::vector<Task>& out) {
  constexpr int kMinPiece = 2, kTries = 400;
  double total = 0.0;
  for (const auto& c : cols) total += c.nz;
  const size_t first = out.size();
  double share = std::max(std::max(total / slots, (double)kMinPiece) + ovh, (total + ovh * cols.size()) / slots);
  int it = 0;
  for (; it < kTries; ++it, share += std::max(0.25, share / 128.0)) {
    out.resize(first);
    int used = 1;
    double left = share;
    for (const auto& c : cols) {
      for (int z = 0; z < c.nz;) {
        if (left < ovh + std::min(kMinPiece, c.nz - z)) {
          ++used;
          left = share;
        }
        int n = std::min(c.nz - z, std::max(kMinPiece, (int)(left - ovh)));
        const int rest = c.nz - z - n;
        if (rest > 0 && rest < kMinPiece) n += n >= 2 * kMinPiece - rest ? rest - kMinPiece : rest;
        out.push_back({c.blk, c.x0, c.y0, z, z + n, 0});
        z += n;
        left -= n + ovh;
      }
      if (used > slots && it + 1 < kTries) break;  // does not fit: a larger share
    }
    if (used <= slots) break;
  }
  return {share, it + 1};
}

// The tasks of a group's columns on `slots` resident CTAs, in the precision form
// prec (0 exact FP64, 1 FP64, 2 FP32).
inline void split_columns(const std::vector<ZColumn>& cols, int slots, int prec, double ovh, std::vector<Task>& out) {
  const size_t first = out.size();
  double share = even_split(cols, slots, ovh, out).share;
  // One round of shares is best (two: vortex 128^3 FP64 841 -> 870 us, 61x83x47
  // blast 131 -> 142, 64x64x256 404 -> 439, 160^3 FP32 1009 -> 1035, vortex 64^3
  // exact 440 -> 495) until the FP64 forms' shares are so long that the CTAs
  // drift apart by more than a second piece's warm-up costs: 64 planes
  // (published form 160^3 2009 -> 1964, 192^3 3442 -> 3229, 256^3 5632 -> 5408;
  // reference form 192^3 2729 -> 2631), 16 in the exact form, whose planes take
  // three times as long (vortex 100^3 2039 -> 1897, 128^3 2734 -> 2693). Three
  // rounds: 256^3 5320, but 192^3 3349 and 128^3 exact 2846. Where the columns
  // outnumber the CTAs a share spans several of them and the second split only
  // adds cuts: no difference beyond 1 % either way (64 blocks of 32 to 95 cells
  // a side, FP64, 3867 -> 3863; exact, 24 to 64, 8703 -> 8606; 256^3 reference
  // form 4252 -> 4280).
  if (prec != 2 && share >= (prec == 0 ? 16.0 : 64.0)) {
    out.resize(first);
    share = even_split(cols, 2 * slots, ovh, out).share;
  }
  // The FP32 form reads its tile halos at a third of the HBM rate, so it
  // gains from neighbouring columns marching in step (their halos meet in
  // L2): equal chunks that fit one round and come within 8 % of the even
  // share replace it (Taylor-Green 110^3 608 -> 592 us, 90^3 vortex 338 ->
  // 332). The FP64 forms do not notice (112^3 blast 374 even, 412 chunked).
  if (prec == 2) {
    int64_t nz = 0;
    for (const auto& c : cols) nz = std::max<int64_t>(nz, c.nz);
    int64_t L = std::max<int64_t>(4, (int64_t)share - 1);
    for (; L <= nz && (double)L + ovh <= 1.08 * share; ++L) {
      int64_t n = 0;
      for (const auto& c : cols) n += (c.nz + L - 1) / L;
      if (n > slots) continue;
      out.resize(first);
      chunk_columns(cols, L, out);
      break;
    }
  }
}

}  // namespace fvm
