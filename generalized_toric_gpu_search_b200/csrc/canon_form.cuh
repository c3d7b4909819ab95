// AGL2(F7) canonical mask of an exponent set: the smallest 49-bit mask among
// the images g(S), g in AGL2(F7), that contain the origin.
//
// The maps are walked by the rows of the image instead of by matrices.  A map
// is chosen by
//   * a direction d, one of the 8 parallel classes of lines of Z_7^2: the rows
//     of the image are the 7 lines of that class;
//   * the line l6 that becomes row 6 and the step dl = 1..6 to the line of the
//     next lower row (row r is line l6 + (6 - r) dl);
//   * a column scale mu = 1..6, and a column shift nu + sigma r of row r.
// The mask is compared from row 6 down, so a candidate is decided by its top
// rows.  A row that is neither empty nor full has one shift that makes it
// smallest (7 is prime), and any shift of a row r >= 1 can be combined with
// any nu (sigma follows), so the top rows of the minimum are those of
// the smallest patterns up to scale and shift: stage 1 keeps, row by row, the
// (d, l6, dl) whose line has the smallest such pattern (a 128-entry table),
// until a row p is reached that is neither empty nor full.  That row fixes
// mu up to its stabiliser and one relation between nu and sigma; the origin
// must be a point of the image, so nu runs over the points of row 0's line.
// Stage 2 evaluates what is left, a few dozen to a few hundred images (about
// 150 on average over 1 to 49 points) instead of 2016 |S|.
//
// Eight lanes serve one set, one direction each in stage 1; the candidates of
// stage 2 of a warp's four sets are dealt out to its lanes through one list in
// shared memory, since most directions keep none and the sets keep uneven
// numbers (dealt out within each set's eight lanes, 9.8 of a warp's 32 lanes
// were active per instruction).  Integer work on registers and small tables: no
// memory traffic but the masks.  1,000,000 sets of 5 to 30 points on a B200:
// 51.5 ms over all 2016 matrices, 3.11 ms this way with a list per set, 2.12
// with one per warp; 50,000 sets of 9 points: 487, 71 and 60 us.
#pragma once

#include "common.cuh"

namespace tg {

// Patterns are 7-bit rows.  `canon` is the smallest pattern over the 42 maps
// x -> mu x + s of Z_7, `mus` the scales that reach it (bit mu - 1).
// scale[mu * 128 + p] is p scaled by mu with, above bit 8, the shift that
// makes it smallest (0 for the empty and the full row).  spread[p] moves bit
// b to bit 7 b.
struct CanonTable {
  uint64_t spread[128];
  uint16_t scale[7 * 128];
  uint8_t canon[128];
  uint8_t mus[128];
};

__host__ __device__ constexpr uint32_t rot7(uint32_t p, int s) {  // p < 128, s in 0..6
  return ((p * 129u) >> (7 - s)) & 127u;
}

constexpr CanonTable make_canon_table() {
  CanonTable t{};
  for (int p = 0; p < 128; ++p) {
    uint32_t best = 127u, mus = 0u;
    for (int mu = 1; mu < 7; ++mu) {
      uint32_t q = 0u;
      for (int b = 0; b < 7; ++b)
        if (p >> b & 1) q |= 1u << (mu * b % 7);
      int s0 = 0;
      for (int s = 1; s < 7; ++s)
        if (rot7(q, s) < rot7(q, s0)) s0 = s;
      t.scale[mu * 128 + p] = uint16_t(q | (uint32_t(s0) << 8));
      const uint32_t v = rot7(q, s0);
      if (v < best) {
        best = v;
        mus = 0u;
      }
      if (v == best) mus |= 1u << (mu - 1);
    }
    t.canon[p] = uint8_t(best);
    t.mus[p] = uint8_t(mus);
    for (int b = 0; b < 7; ++b)
      if (p >> b & 1) t.spread[p] |= 1ull << (7 * b);
  }
  return t;
}

__device__ const CanonTable g_canon_table = make_canon_table();

constexpr int kCanonItems = 256;  // candidates listed at a time, per warp

struct CanonScratch {  // shared memory of one warp (four sets)
  uint64_t img[32];             // the sets seen from each direction: row l = line l
  uint64_t prefix[4];
  unsigned long long best[4];
  int p[4];
  uint16_t item[kCanonItems];
};

__device__ __forceinline__ int mod7(int x) { return x >= 7 ? x - 7 : x; }  // x < 14

// The canonical masks of the four sets of a warp (group = lane / 8; the lanes
// of a group pass the same S, all the same scratch; S = 0 returns ~0).  The whole warp
// calls it: loops run until the last group is done, so every shuffle and
// vote is warp-wide.
__device__ __forceinline__ uint64_t canon_mask_groups(int lane, uint64_t S, const CanonTable& T,
                                                      CanonScratch& sc) {
  const int d = lane & 7, group = lane >> 3;
  // Direction 7: rows as they are.  Direction m < 7: point (a, b) lies on
  // line b + m a at column a.
  uint64_t img = 0ull;
  if (d == 7) {
    img = S;
  } else {
    for (int a = 0, s = 0; a < 7; ++a, s = mod7(s + d))
      img |= T.spread[rot7(uint32_t(S >> (7 * a)) & 127u, s)] << a;
  }
  __syncwarp();
  sc.img[lane] = img;

  // Candidates (l6, dl) of this direction, bit 6 l6 + dl - 1: the line of row
  // 0, l6 - dl, must hold a point.  Row 6 is decided with them.
  uint64_t cand = 0ull;
  uint32_t vmin = 255u;
  {
    uint32_t nz = 0u;
    for (int l = 0; l < 7; ++l) nz |= ((uint32_t(img >> (7 * l)) & 127u) != 0u ? 1u : 0u) << l;
    const uint32_t rev = __brev(nz) >> 25;
    for (int l = 0; l < 7; ++l) {
      // bit dl - 1 is line l - dl
      const uint32_t f = ((rev << l) | (rev >> (7 - l))) & 63u;
      const uint32_t v = T.canon[uint32_t(img >> (7 * l)) & 127u];
      if (f != 0u && v <= vmin) {
        if (v < vmin) cand = 0ull;
        vmin = v;
        cand |= uint64_t(f) << (6 * l);
      }
    }
  }
  // Rows 6, 5, ... until one is neither empty nor full (p, 0 when none is).
  uint64_t prefix = 0ull;  // rows 6..p of the minimum
  int p = 0;
  bool open = true;
  for (int r = 6;;) {
    uint32_t v = vmin;
    for (int o = 4; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (open) {
      if (vmin != v) cand = 0ull;
      prefix = (prefix << 7) | v;
      if (v != 0u && v != 127u) {
        p = r;
        open = false;
      }
    }
    if (--r == 0 || !__any_sync(0xffffffffu, open)) break;
    if (open) {
      vmin = 255u;
      uint64_t keep = 0ull;
      for (uint64_t x = cand; x != 0ull; x &= x - 1ull) {
        const int bit = __ffsll(static_cast<long long>(x)) - 1;
        const int l6 = bit / 6, dl = bit - 6 * l6 + 1;
        const uint32_t c = T.canon[uint32_t(img >> (7 * ((l6 + (6 - r) * dl) % 7))) & 127u];
        if (c <= vmin) {
          if (c < vmin) keep = 0ull;
          vmin = c;
          keep |= 1ull << bit;
        }
      }
      cand = keep;
    }
  }

  // Every map fixes the full set, and all its 2016 candidates would tie: 100
  // such sets take 80 us a call without them, 1011 with.
  const bool whole = S == kMask49;
  if (whole) cand = 0ull;

  // Stage 2: (group, d, l6, dl, mu) of the kept candidates, listed for the warp.
  int mine = 0;
  for (uint64_t x = cand; x != 0ull; x &= x - 1ull) {
    const int bit = __ffsll(static_cast<long long>(x)) - 1;
    const int l6 = bit / 6, dl = bit - 6 * l6 + 1;
    const uint32_t pat = uint32_t(img >> (7 * ((l6 + (6 - p) * dl) % 7))) & 127u;
    mine += p ? __popc(T.mus[pat]) : 6;
  }
  int end = mine;  // inclusive prefix over the warp
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end += y;
  }
  const int total = __shfl_sync(0xffffffffu, end, 31);
  const int begin = end - mine;
  if (d == 0) {
    sc.prefix[group] = prefix;
    sc.p[group] = p;
    sc.best[group] = whole ? S : ~0ull;
  }
  for (int base = 0; base < total; base += kCanonItems) {
    __syncwarp();
    int at = begin - base;
    for (uint64_t x = cand; x != 0ull; x &= x - 1ull) {
      const int bit = __ffsll(static_cast<long long>(x)) - 1;
      const int l6 = bit / 6, dl = bit - 6 * l6 + 1;
      const uint32_t pat = uint32_t(img >> (7 * ((l6 + (6 - p) * dl) % 7))) & 127u;
      for (uint32_t m = p ? uint32_t(T.mus[pat]) : 63u; m != 0u; m &= m - 1u, ++at)
        if (at >= 0 && at < kCanonItems)
          sc.item[at] = uint16_t(d | (l6 << 3) | (dl << 6) | (__ffs(int(m)) << 9) | (group << 12));
    }
    __syncwarp();
    const int n = min(kCanonItems, total - base);
    for (int i = lane; i < n; i += 32) {
      const uint32_t it = sc.item[i];
      const uint32_t of = it >> 12;
      const uint64_t g = sc.img[8u * of + (it & 7u)], pre = sc.prefix[of];
      const int q = sc.p[of], dl = int(it >> 6) & 7;
      const int inv_q = (0x6325410 >> (4 * q)) & 7;  // 1 / q mod 7 (0 for q = 0)
      const int top = q > 0 ? q - 1 : 0;             // first row stage 2 decides
      const uint16_t* scale = T.scale + ((it >> 9) & 7u) * 128u;
      int line = (int(it >> 3 & 7u) + (6 - q) * dl) % 7;
      const int rho = q ? scale[uint32_t(g >> (7 * line)) & 127u] >> 8 : 0;
      uint64_t rows = 0ull;  // scaled rows top..0
      if (q) line = mod7(line + dl);
      else line = mod7(int(it >> 3 & 7u) + 7 - dl);  // row 0
      for (int r = top; r >= 0; --r) {
        rows = (rows << 7) | (scale[uint32_t(g >> (7 * line)) & 127u] & 127u);
        line = mod7(line + dl);
      }
      // what any lane has reached for this set (a late look only prunes less)
      const uint64_t seen = *reinterpret_cast<volatile unsigned long long*>(&sc.best[of]);
      uint64_t best = seen;
      for (uint32_t pts = uint32_t(rows) & 127u; pts != 0u; pts &= pts - 1u) {
        const int nu = mod7(8 - __ffs(int(pts)));  // moves the point to column 0
        const int neg = q ? ((nu + 7 - rho) * inv_q) % 7 : 0;  // -sigma
        int s = q ? mod7(rho + neg) : nu;
        uint64_t cur = (pre << 7) | rot7(uint32_t(rows >> (7 * top)) & 127u, s);
        if (cur > (best >> (7 * top))) continue;
        for (int r = top - 1; r >= 0; --r) {
          s = mod7(s + neg);
          cur = (cur << 7) | rot7(uint32_t(rows >> (7 * r)) & 127u, s);
        }
        best = cur < best ? cur : best;
      }
      if (best < seen) atomicMin(&sc.best[of], static_cast<unsigned long long>(best));
    }
  }
  __syncwarp();
  return sc.best[group];
}

}  // namespace tg
