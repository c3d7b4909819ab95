// Minimum distance of toric codes by information sets.  Included by
// distance.cu, whose tables, descriptors and helpers it shares.
//
// What is enumerated.  A code's generator is reduced to the identity on one
// information set E of k columns; the torus translations permute the 49
// columns regularly and map the code onto itself, so every translate of E is
// an information set with the same messages.  After all messages of weight
// <= L on E, a codeword not met weighs at least ceil(49 (L + 1) / k) (it
// weighs L + 1 on every translate, and each column lies in k of them).  Two
// parts of level w = L + 1 raise that bound before the level is complete:
//   * the supports holding the last row:  ceil(49 w / (k - 1))
//     (infoset_kernel.cuh, is_split_level);
//   * the supports avoiding the last r rows A:  ceil(49 (w + 1) / (k + r)).
//     A codeword not met weighs w on every translate, and w + 1 on each one
//     whose restriction avoids A; at least 49 - r wt of them do (each column
//     of A is hit by wt translates), so k wt >= 49 w + 49 - r wt.
// tw_next picks, from the best weight so far, the cheapest part that settles
// the code, else the next whole level.
//
// How.  The codeword of a support of w rows is split: u takes the w - 2
// largest rows (the smallest of them, the pivot row p, with coefficient 1), v
// the two rows below p.  The pairs v of one code, in colexicographic order,
// are the same for every u but for their number (49 C(p, 2)), so they are laid
// out once in shared memory by columns: for each counted column and each of
// the eight field values, one bit per pair that has the value there.  The bit
// row that u's value selects says which pairs make a zero in that column, and
// a carry-save adder over the columns' rows counts the zeros of 32 codewords
// at once.  30 columns cost 30 words of shared memory and 54 LOP3 per 32
// codewords and lane; a POPC per codeword costs 5 ALU operations each and two
// cycles of the POPC pipe per warp.  A part of the 49 - k columns outside E is
// enough: a codeword lighter than the best so far has few nonzeros, and the
// rare ones that pass are weighed whole.
//
// The bounds are the ALU (31 codewords per cycle and SM) and shared memory
// (128 bytes a cycle: 34).  Whole launches reach 17 to 19 from k = 14 on, 15.5
// at k = 13, 12 at k = 12 (more columns, shorter lists) and 15 over 10,000 sets
// of k = 6..14, against 10 of the walk by POPC (infoset_kernel.cuh).  At
// k = 14 (1,000 sets, 17) the ALU is 80 % busy and the shared-memory pipe 72 %:
// pairs past the end of a lane's list, the build and the batches' own work take
// what the bound leaves.  The same sums as a contraction of +-1 characters on
// tcgen05 were slower: a unit's handovers cost the short lists more than the
// sums.
//
// Kernels.  toric_prep_kernel: one CTA per code, elimination, tables, levels
// 1 to 3 (level 4 of short codes), first stage.  toric_walk_kernel: two
// persistent CTAs per SM; codes move through their stages on their own (the
// CTA that counts a stage's last claim opens the next one), so no launch and
// no barrier separates the levels.  One set of k = 8 takes 54 us by the Python
// call (180 by the general walk's 31 launches), of k = 14 122 (304), 10,000
// sets of k = 6..14 3.1 ms (4.25).
#pragma once

namespace tg {

// ---------------------------------------------------------------------------
// Geometry
// ---------------------------------------------------------------------------

// Bit rows of a CTA: columns times words of 32 pairs.  Codes of up to 12 rows
// have many columns outside E and large distances, so 32 columns let too many
// codewords pass (a few percent at k = 8), but few pairs; the others have pairs
// enough for most of their u's in one block.  Either layout leaves room for two
// CTAs on an SM (one builds or waits for work while the other counts).
// Four words of a column and value lie together (one 16-byte load), the eight
// values next to each other: the lanes of a load read one 128-byte row.  The
// odd 16 bytes keep the columns' rows in different banks while they are built.
template <int kColsT, int kWordsT>
struct TwLayoutOf {
  static constexpr int kCols = kColsT, kWords = kWordsT, kPairs = 32 * kWordsT;
  static constexpr int kColBytes = kWordsT / 4 * 128 + 16;
  static constexpr int kRowBytes = kColsT <= 32 ? 32 : 48;  // a row's value offsets
  static constexpr int kTableBytes = kColsT * kColBytes;
  static_assert(kWordsT % 8 == 0, "two groups of words at a time");
};
using TwWide = TwLayoutOf<42, 72>;     // k <= 12: at most 2205 pairs
using TwNarrow = TwLayoutOf<32, 104>;  // 3328 pairs
constexpr int kTwWideK = 12;
constexpr int kTwThreads = 256, kTwWarps = kTwThreads / 32;
constexpr int kTwCtasPerSm = 2;
constexpr int kTwWideBytes = TwWide::kTableBytes + kTwWideK * 7 * TwWide::kRowBytes;
constexpr int kTwNarrowBytes = TwNarrow::kTableBytes + kMaxExactK * 7 * TwNarrow::kRowBytes;
constexpr int kTwSharedBytes = kTwWideBytes > kTwNarrowBytes ? kTwWideBytes : kTwNarrowBytes;

__host__ __device__ constexpr uint32_t tw_pairs(int k) {
  return k <= kTwWideK ? TwWide::kPairs : TwNarrow::kPairs;
}

// Picks of b of 21 rows, b = 1..4, in colexicographic order (the picks of
// rows < n are the first C(n, b)): 5 bits per row.
constexpr int kTwCombs = 21 + 210 + 1330 + 5985;
__device__ uint32_t g_tw_comb[kTwCombs];

// Where the picks of b rows begin.
__device__ __forceinline__ int tw_comb_off(int b) {
  return b == 1 ? 0 : b == 2 ? 21 : b == 3 ? 231 : 1561;
}

// ---------------------------------------------------------------------------
// Queue and per-code state (in the workspace's information-set region)
// ---------------------------------------------------------------------------

struct TwHeader {
  unsigned int head;  // places drawn
  unsigned int pad0[31];
  unsigned int tail;  // tickets put in
  unsigned int pad1[31];
  int open;           // codes with a stage under way
  unsigned int pad2[31];
  unsigned int progress;  // counted up as work ends
  unsigned int pad3[31];
};

// One stage of a code: the supports of w rows, without the last `part` rows
// (part <= 3) or with the last row in each (kTwForced), against one block of
// pairs.
constexpr int kTwForced = 4;
struct TwStage {
  int8_t w, part, block;
  int8_t cut;  // the pairs of a batch are cut into 2^cut pieces
  __device__ int avoid() const { return part < kTwForced ? part : 0; }
  __device__ int forced() const { return part == kTwForced ? 1 : 0; }
};

// Work on a stage is claimed in pieces of batches of 32 u's (or several, so
// that a 32-bit number suffices): claim i takes pieces i, i + claims, ... .
struct __align__(16) TwState {
  // read together (tw_look): the stage number is written before anything else
  // of a new stage, the claim counter last
  unsigned long long claim;  // stage number << 32 | next claim
  unsigned int claims;       // claims of the stage
  unsigned int done;         // claims done
  unsigned int seq;          // stage number
  TwStage stage;
  int level;                 // once the stage is done: all supports of at most `level` rows are
                             // met; 64: and those of level + 1 that hold the last row
  int tickets;               // of this code in the queue
};
static_assert(sizeof(TwState) == 32, "TwState");

struct TwLayout {
  size_t queue, state, tab, rows, end;
  unsigned int cap;
};

// The region: TwHeader, queue (cleared with it), states, tables, rows; about
// 3,100 bytes per code at k_max = 21.  The queue is a ring: in a big batch a
// code has one ticket in it, and each CTA may be about to add up to 16.
__host__ __device__ inline TwLayout tw_layout(int n, int k_max) {
  TwLayout L;
  const size_t state = size_t(n) * sizeof(TwState);
  const size_t tab = size_t(n) * k_max * 7 * 16;
  const size_t rows = size_t(n) * k_max * sizeof(V6);
  L.cap = (static_cast<unsigned int>(2 * n) + 8192u + 7u) & ~7u;
  L.queue = sizeof(TwHeader);
  L.state = L.queue + size_t(L.cap) * 4;
  L.tab = L.state + state;
  L.rows = L.tab + tab;
  L.end = L.rows + rows;
  return L;
}

__device__ __forceinline__ unsigned int tw_ld_acquire(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void tw_st_release(unsigned int* p, unsigned int v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ---------------------------------------------------------------------------
// Stages
// ---------------------------------------------------------------------------

__device__ __forceinline__ int tw_ceil_div(int a, int b) { return (a + b - 1) / b; }

// The next stage of a k-row code whose messages up to weight `level` are met
// (and, when p1, those of weight level + 1 that hold the last row), with best
// weight `best` and target distance `wthr`.  Returns false when the code is
// settled.  `level` and `p1` become what holds once that stage is done; a
// part that settles the code whatever comes of it (`best` only falls) counts
// as the last level.
__device__ inline bool tw_next(int k, int best, int wthr, int& level, bool& p1, TwStage& st) {
  if (best < wthr || level >= k) return false;
  if (tw_ceil_div(kN * (level + 1), k) >= best) return false;
  const int w = level + 1;
  if (p1 && tw_ceil_div(kN * w, k - 1) >= best) return false;
  // the largest set of avoided rows that still settles the code (-1: not
  // even the whole level does)
  int avoid = -1;
  while (avoid < 3 && k - (avoid + 1) >= w &&
         tw_ceil_div(kN * (w + 1), k + avoid + 1) >= best)
    ++avoid;
  const bool last_row = !p1 && tw_ceil_div(kN * w, k - 1) >= best;
  st = TwStage{};
  st.w = int8_t(w);
  if ((last_row && (avoid < 0 || c_binom[k - 1][w - 1] <= c_binom[k - avoid][w])) ||
      (!p1 && w > 4 && avoid < 0)) {
    // the part settles the code, or more levels are to come: half now, then
    // look again
    st.part = kTwForced;
    p1 = true;
    return true;
  }
  if (avoid > 0 || p1) {  // after part 1, the rest is what avoids the last row
    st.part = int8_t(avoid > 1 ? avoid : 1);
    level = avoid > 0 ? k : w;
    p1 = false;
    return true;
  }
  level = w;
  return true;
}

// The weight at which a code under this stage is decided: below the target, or
// what the levels before it prove.
__device__ __forceinline__ int tw_stop(int k, const TwStage& st, int wthr) {
  return max(wthr - 1, tw_ceil_div(kN * st.w, k));
}

// Pairs below pivot row p.
__device__ __forceinline__ uint32_t tw_pairs_below(int p) {
  return 49u * static_cast<uint32_t>(p * (p - 1) / 2);
}

// u's of pivot row p in the stage.
__device__ __forceinline__ unsigned long long tw_us(int k, const TwStage& st, int p) {
  const int rows = k - st.avoid() - 1 - p - st.forced(), picks = st.w - 3 - st.forced();
  return rows >= picks && p >= 2 ? c_binom[rows][picks] * c_pow7[st.w - 3] : 0ull;
}

struct TwView {  // the region's arrays
  TwHeader* hdr;
  unsigned int* queue;
  TwState* state;
  uint4* tab;
  V6* rows;
  unsigned int cap;
};

__device__ __forceinline__ TwView tw_view(const DistArgs& a) {
  uint8_t* b = reinterpret_cast<uint8_t*>(a.is_rows);
  const TwLayout L = tw_layout(a.n, a.k_max);
  return TwView{reinterpret_cast<TwHeader*>(b), reinterpret_cast<unsigned int*>(b + L.queue),
                reinterpret_cast<TwState*>(b + L.state), reinterpret_cast<uint4*>(b + L.tab),
                reinterpret_cast<V6*>(b + L.rows), L.cap};
}

// Each lane gets the number of u's up to and with pivot row `lane` that have
// pairs in the stage's block; `words` the stage's codewords.
__device__ __forceinline__ unsigned long long tw_ends(int k, const TwStage& st, int lane,
                                                      unsigned long long& words) {
  unsigned long long end = lane < k ? tw_us(k, st, lane) : 0ull;
  const uint32_t first = static_cast<uint32_t>(st.block) * tw_pairs(k);
  const uint32_t nv = end && tw_pairs_below(lane) > first ? tw_pairs_below(lane) - first : 0u;
  if (nv == 0u) end = 0ull;
  words = end * min(nv, tw_pairs(k));
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end += y;
  }
  for (int o = 16; o > 0; o >>= 1) words += __shfl_xor_sync(0xffffffffu, words, o);
  return end;
}

// Claims of a stage to aim at: two for each warp of the CTAs that may work on
// it.
constexpr int kTwClaims = 2 * kTwWarps;

// In place of a ticket: no code is open any more.
constexpr unsigned int kTwOver = 0xFFFFFFFFu;

// CTAs that wait for a ticket, up to 16.
__device__ __forceinline__ int tw_waiting(const TwView& v) {
  const unsigned int head = *reinterpret_cast<volatile unsigned int*>(&v.hdr->head);
  const unsigned int tail = *reinterpret_cast<volatile unsigned int*>(&v.hdr->tail);
  return min(max(int(head - tail), 0), 16);
}

// Puts tickets of code c into the queue, up to `want` less those that are there
// (one whole warp; `want` counts in lane 0).
__device__ __forceinline__ void tw_push(const DistArgs& a, const TwView& v, int lane, int c,
                                        int want) {
  int count = 0;
  unsigned int pos = 0u;
  if (lane == 0) {
    count = want - atomicAdd(&v.state[c].tickets, 0);
    if (count > 0) {
      atomicAdd(&v.state[c].tickets, count);
      pos = atomicAdd(&v.hdr->tail, static_cast<unsigned int>(count));
    }
  }
  count = __shfl_sync(0xffffffffu, count, 0);
  pos = __shfl_sync(0xffffffffu, pos, 0);
  for (int i = lane; i < count; i += 32) {
    unsigned int* slot = v.queue + (pos + i) % v.cap;
    // free, unless a whole ring of tickets has overtaken the CTA that draws it,
    // or all codes are settled
    for (int tries = 0;; ++tries) {
      const unsigned int old = atomicCAS(slot, 0u, static_cast<unsigned int>(c) + 1u);
      if (old == 0u || old == kTwOver) break;
      if (tries == 1 << 22) {
        report_status(a.hdr, TG_ERR_STATE);
        break;
      }
    }
  }
  __syncwarp();
}

// Tells every CTA that waits or will wait that no code is open (one whole warp).
__device__ __forceinline__ void tw_over(const DistArgs& a, const TwView& v, int lane) {
  const unsigned int tail = *reinterpret_cast<volatile unsigned int*>(&v.hdr->tail);
  for (int i = lane; i < a.tw_ctas; i += 32)
    *reinterpret_cast<volatile unsigned int*>(v.queue + (tail + i) % v.cap) = kTwOver;
  __syncwarp();
}

// Settles code c or opens its next stage, with everything before it done.
// Called by one whole warp; `open` counts the code in (first call) or out.
__device__ inline void tw_advance(const DistArgs& a, const TwView& v, int lane, int c, int k,
                                  int level, bool p1, TwStage st, unsigned int seq, bool first) {
  const int best = __shfl_sync(0xffffffffu, ld_flag(a.is_best + c), 0);
  const int wthr = kN - a.desc[c].tmax;
  unsigned long long words = 0ull, total = 0ull;
  if (!first && best > tw_stop(k, st, wthr)) {
    // the stage's next block of pairs, if there is one
    ++st.block;
    total = __shfl_sync(0xffffffffu, tw_ends(k, st, lane, words), 31);
  }
  if (total == 0ull) {
    if (!tw_next(k, best, wthr, level, p1, st)) {
      int open = 1;
      if (lane == 0) {
        a.out[c] = kN - best;
        a.abort[c] = 1;
        __threadfence();
        if (!first) open = atomicSub(&v.hdr->open, 1) - 1;
      }
      if (__shfl_sync(0xffffffffu, open, 0) == 0) tw_over(a, v, lane);
      return;
    }
    total = __shfl_sync(0xffffffffu, tw_ends(k, st, lane, words), 31);
  }
  total = (total + 31ull) / 32ull;
  const int share = tw_ceil_div(a.tw_ctas, a.n);  // CTAs per code
  const unsigned long long aim = static_cast<unsigned long long>(kTwClaims * share);
  st.cut = 0;
  while (st.cut < 3 && total < aim) {
    ++st.cut;
    total *= 2ull;
  }
  const unsigned long long per = (total >> 28) + 1ull;
  const unsigned int claims = static_cast<unsigned int>((total + per - 1ull) / per);
  int want = 0;
  if (lane == 0) {
    // the stage number first: a reader that finds the old one before and after
    // its look has seen the old stage
    volatile TwState& s = v.state[c];
    s.seq = seq;
    __threadfence();
    s.done = 0u;
    s.claims = claims;
    s.level = level | (p1 ? 64 : 0);
    v.state[c].stage = st;
    if (first) s.tickets = 0;
    __threadfence();
    atomicExch(&v.state[c].claim, static_cast<unsigned long long>(seq) << 32);
    if (first) atomicAdd(&v.hdr->open, 1);
    atomicAdd(&a.is_hdr->tasks_all, total);
    // Tickets for as many CTAs as keep the chip busy.  Those still in the queue
    // serve the new stage, too: whoever draws one counts it out before looking
    // at the stage, and here it is counted after the stage is open.
    __threadfence();
    want = min(min(max(share, tw_waiting(v)), 64), int((claims + kTwWarps - 1) / kTwWarps));
  }
  tw_push(a, v, lane, c, want);
}

// ---------------------------------------------------------------------------
// Preparation
// ---------------------------------------------------------------------------

constexpr int kTwPrepThreads = 128;

// One word's columns of a vector (three planes).
struct TwCols {
  uint32_t x0, x1, x2;
};

__device__ __forceinline__ TwCols tw_alpha(const TwCols& g) {
  return TwCols{g.x2, g.x0 ^ g.x2, g.x1};
}

__device__ __forceinline__ TwCols tw_sum(const TwCols& a, const TwCols& b) {
  return TwCols{a.x0 ^ b.x0, a.x1 ^ b.x1, a.x2 ^ b.x2};
}

__device__ __forceinline__ TwCols tw_mul(const TwCols& a, const TwCols& b) {
  const uint32_t d3 = (a.x1 & b.x2) ^ (a.x2 & b.x1), d4 = a.x2 & b.x2;
  return TwCols{(a.x0 & b.x0) ^ d3, (a.x0 & b.x1) ^ (a.x1 & b.x0) ^ d3 ^ d4,
                (a.x0 & b.x2) ^ (a.x1 & b.x1) ^ (a.x2 & b.x0) ^ d4};
}

// a / b column by column, a itself where b is 0, and the columns where b is
// not.  1 / b = b^2 b^4; squares are linear.
__device__ __forceinline__ uint4 tw_ratio(const TwCols& a, TwCols b) {
  const uint32_t nz = b.x0 | b.x1 | b.x2;
  b.x0 |= ~nz;
  const TwCols b2{b.x0, b.x2, b.x1 ^ b.x2};
  const TwCols b4{b2.x0, b2.x2, b2.x1 ^ b2.x2};
  const TwCols w = tw_mul(a, tw_mul(b2, b4));
  return make_uint4(w.x0, w.x1, w.x2, nz);
}

// Sweeps over the last coefficient: the seven codewords P + alpha^v Z, from
// P / Z.  A column of it names the v that makes a zero there, so a codeword and
// word of columns take one LOP3 and one POPC (by planes of P + alpha^v Z three
// and one, which bound the sweep by the ALU); where Z is 0 the column is P's
// own.  Row r / row z for all r < z is laid out once per code.
// Whole calls: 4,000 sets of k = 8 237 -> 201 us, of k = 10 515 -> 454, 39,000
// of k = 10 3.93 -> 3.40 ms, 10,000 of k = 6..14 2.95 -> 2.80; a lone set the
// same.
struct TwRatio {
  uint4 lo, hi;
};

__device__ __forceinline__ TwCols tw_cols(const uint4& w) { return TwCols{w.x, w.y, w.z}; }

// The columns where P + alpha^v Z is not 0 for any v, or only for one v.
__device__ __forceinline__ int tw_own(const TwCols& g, uint32_t nz) {
  return __popc(lop3<0xFE>(g.x0, g.x1, g.x2) | nz);
}

__device__ __forceinline__ TwCols tw_mask(const TwCols& g, uint32_t nz) {
  return TwCols{g.x0 & nz, g.x1 & nz, g.x2 & nz};
}

// Most zeros that one v makes (g masked).
__device__ __forceinline__ int tw_most(const TwCols& g) {
  int most = __popc(lop3<sel_lut(1)>(g.x0, g.x1, g.x2));
  most = max(most, __popc(lop3<sel_lut(2)>(g.x0, g.x1, g.x2)));
  most = max(most, __popc(lop3<sel_lut(3)>(g.x0, g.x1, g.x2)));
  most = max(most, __popc(lop3<sel_lut(4)>(g.x0, g.x1, g.x2)));
  most = max(most, __popc(lop3<sel_lut(5)>(g.x0, g.x1, g.x2)));
  most = max(most, __popc(lop3<sel_lut(6)>(g.x0, g.x1, g.x2)));
  return max(most, __popc(lop3<sel_lut(7)>(g.x0, g.x1, g.x2)));
}

template <int kV>
__device__ __forceinline__ int tw_zeros(const TwCols& g, const TwCols& h) {
  return __popc(lop3<sel_lut(kV)>(g.x0, g.x1, g.x2)) + __popc(lop3<sel_lut(kV)>(h.x0, h.x1, h.x2));
}

// Least weight over all columns.
__device__ __forceinline__ int tw_least(const TwCols& lo, const TwCols& hi, uint32_t nz_lo,
                                        uint32_t nz_hi) {
  const TwCols g = tw_mask(lo, nz_lo), h = tw_mask(hi, nz_hi);
  int most = tw_zeros<1>(g, h);
  most = max(most, tw_zeros<2>(g, h));
  most = max(most, tw_zeros<3>(g, h));
  most = max(most, tw_zeros<4>(g, h));
  most = max(most, tw_zeros<5>(g, h));
  most = max(most, tw_zeros<6>(g, h));
  most = max(most, tw_zeros<7>(g, h));
  return tw_own(lo, nz_lo) + tw_own(hi, nz_hi) - most;
}

// Codes of at most this many rows have their level 4 done by toric_prep_kernel
// (1.7e5 codewords at k = 12, 3.4e5 at k = 14), for which the walk's bit rows
// and its round trips cost more than the codewords: 10,000 sets of k = 6..14
// 3.13 ms up to 13, 2.89 up to 14, 2.90 up to 16.  A lone code of k = 14 is
// better off with all CTAs on it (0.13 ms, 0.15), so the limit is lower where
// the codes do not fill the chip (11: 40 sets of k = 14 0.225 ms, 12: 0.203).
constexpr int kTwPrepK = 12, kTwPrepKBig = 14;

// Up to this many rows level 4 counts all columns at once.  The best weights of
// short codes let too many sweeps past the first 32 columns, whose second count
// holds up the warp; from 11 rows on few pass.  4,000 sets: k = 9 282 us by the
// first columns, 257 whole; k = 10 476 and 455; k = 11 1095 and 1116.
constexpr int kTwWholeK = 10;

// Least weight, below wmin, of the codewords of a stage of level 4: seven
// sweeps a unit.  kWhole: all columns are counted.  Else the first 32 and the 4
// on E rule out most, and what they leave is counted whole after the sweeps.
template <bool kWhole>
__device__ __forceinline__ int tw_level4(const TwRatio* ratio, int k, const TwStage& st, int wmin,
                                         int stop, int tid) {
  const int picks = 4 - st.forced(), m = k - st.avoid() - st.forced();
  const uint32_t units = 7u * static_cast<uint32_t>(c_binom[m][picks]);
  const auto pick = [&](uint32_t i) {
    return i < units ? __ldg(g_tw_comb + tw_comb_off(picks) + i / 7u) : 0u;
  };
  uint32_t next = pick(tid);
  for (uint32_t i = tid; i < units && wmin > stop; i += kTwPrepThreads) {
    const uint32_t s = i % 7u, r = next;
    next = pick(i + kTwPrepThreads);  // on its way during the sweeps
    const uint32_t rz = picks == 4 ? r >> 15 : uint32_t(k - 1);
    const TwRatio* by_z = ratio + rz * (rz - 1u) / 2u;
    const TwRatio &Q = by_z[r & 31u], &X = by_z[(r >> 5) & 31u], &Y = by_z[(r >> 10) & 31u];
    const uint32_t nz_lo = Q.lo.w, nz_hi = Q.hi.w;
    const auto head = [&](const uint4& q, TwCols x) {
      for (uint32_t e = 0; e < s; ++e) x = tw_alpha(x);
      return tw_sum(tw_cols(q), x);
    };
    const TwCols p = head(Q.lo, tw_cols(X.lo));
    TwCols y = tw_cols(Y.lo);
    if constexpr (kWhole) {
      const TwCols ph = head(Q.hi, tw_cols(X.hi));
      TwCols yh = tw_cols(Y.hi);
#pragma unroll
      for (int t = 0; t < 7; ++t) {
        wmin = min(wmin, tw_least(tw_sum(p, y), tw_sum(ph, yh), nz_lo, nz_hi));
        y = tw_alpha(y);
        yh = tw_alpha(yh);
      }
    } else {
      uint32_t light = 0u;  // bit t: one of the seven codewords may be lighter
#pragma unroll
      for (int t = 0; t < 7; ++t) {
        const TwCols g = tw_sum(p, y);
        if (tw_own(g, nz_lo) - tw_most(tw_mask(g, nz_lo)) + 4 < wmin) light |= 1u << t;
        y = tw_alpha(y);
      }
      if (light) {
        const TwCols ph = head(Q.hi, tw_cols(X.hi));
        TwCols yh = tw_cols(Y.hi);  // y is back at alpha^7 = 1
#pragma unroll 1
        for (; light; light >>= 1) {
          if (light & 1u) wmin = min(wmin, tw_least(tw_sum(p, y), tw_sum(ph, yh), nz_lo, nz_hi));
          y = tw_alpha(y);
          yh = tw_alpha(yh);
        }
      }
    }
  }
  return wmin;
}

__global__ void __launch_bounds__(kTwPrepThreads) toric_prep_kernel(DistArgs a) {
  __shared__ __align__(16) V6 s_rows[kMaxExactK];
  __shared__ TwRatio s_ratio[kMaxExactK * (kMaxExactK - 1) / 2];
  __shared__ int s_min[kTwPrepThreads / 32];
  __shared__ int s_walk;
  const TwView view = tw_view(a);
  const int c = blockIdx.x;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  uint32_t pair = __ldg(g_tw_comb + tw_comb_off(2) + tid);  // here by the end of the elimination
  const int64_t beg = a.off[c];
  const int64_t klong = a.off[c + 1] - beg;
  const bool ok_k = klong >= 0 && klong <= a.k_max;
  const int k = ok_k ? int(klong) : 0;
  if (tid < 32) {
    const int my = lane < k ? a.idx[beg + lane] : 0;
    const bool bad = __any_sync(0xffffffffu, lane < k && (my < 0 || my >= kN)) || !ok_k;
    uint64_t p0 = 0ull, p1 = 0ull, p2 = 0ull;
    if (lane < k && !bad) {
      p0 = __ldg(a.tab.Mp + my * 3);
      p1 = __ldg(a.tab.Mp + my * 3 + 1);
      p2 = __ldg(a.tab.Mp + my * 3 + 2);
    }
    // Gauss-Jordan: row r takes its own first nonzero column as pivot (any
    // information set serves), so no column is searched and no row moves.
    uint64_t used = 0ull;
    bool deficient = false;
    if (!bad && k > 1) {
      for (int r = 0; r < k; ++r) {
        const uint64_t nz = p0 | p1 | p2;
        const int col = __shfl_sync(0xffffffffu, __ffsll(static_cast<long long>(nz)) - 1, r);
        if (col < 0) {
          deficient = true;  // dependent rows: a nonzero message gives the zero codeword
          break;
        }
        const uint32_t coef = uint32_t((p0 >> col) & 1ull) | (uint32_t((p1 >> col) & 1ull) << 1) |
                              (uint32_t((p2 >> col) & 1ull) << 2);
        const uint32_t inv = c_inv[__shfl_sync(0xffffffffu, coef, r)];
        uint64_t q0 = __shfl_sync(0xffffffffu, p0, r);
        uint64_t q1 = __shfl_sync(0xffffffffu, p1, r);
        uint64_t q2 = __shfl_sync(0xffffffffu, p2, r);
        gf8_scale64(lane == r ? inv : c_mul[coef * 8 + inv], q0, q1, q2);
        p0 = lane == r ? q0 : p0 ^ q0;
        p1 = lane == r ? q1 : p1 ^ q1;
        p2 = lane == r ? q2 : p2 ^ q2;
        used |= 1ull << col;
      }
    }
    const bool walk = !bad && k > 1 && !deficient;
    if (lane == 0) {
      CodeDesc d{};
      d.k = k;
      d.R = d.H = 1;
      d.tmax = kN - (a.target ? a.target[c] : a.td_default);
      d.set_id = c;
      d.flags = kIsCodeFlag | kTorusBoundFlag | (walk ? 0 : kDecidedFlag);
      a.desc[c] = d;
      // one row: its own zeros
      const int z = k == 1 ? kN - __popcll((p0 | p1 | p2) & kMask49) : 0;
      a.out[c] = bad ? 0 : deficient ? kN : z;
      a.abort[c] = walk ? 0 : 1;
      if (bad) report_status(a.hdr, TG_ERR_BAD_INPUT);
      if (!bad && k > 0) atomicAdd(&a.hdr->ref_messages, double(pow8(k)) - 1.0);
      s_walk = walk ? 1 : 0;
    }
    if (walk) {
      is_reorder_columns(used, p0, p1, p2);
      if (lane < k) {
        const V6 g = v6_of_planes(p0, p1, p2);
        s_rows[lane] = g;
        v6_stg(view.rows + size_t(c) * a.k_max + lane, g);
        // alpha^e g on the first 42 columns, as far as they lie outside E: three
        // planes of 32, and those of ten more packed in a word
        const int n_red = kN - k;
        const uint32_t m = n_red >= 32 ? ~0u : (1u << n_red) - 1u;
        const uint32_t mh = n_red >= 42 ? 0x3FFu : n_red > 32 ? (1u << (n_red - 32)) - 1u : 0u;
        V6 t = g;
        uint4* dst = view.tab + (size_t(c) * a.k_max + lane) * 7;
        for (int e = 0; e < 7; ++e) {
          dst[e] = make_uint4(t.l0 & m, t.l1 & m, t.l2 & m,
                              (t.h0 & mh) | ((t.h1 & mh) << 10) | ((t.h2 & mh) << 20));
          v6_alpha_pow(t, 1);
        }
      }
    }
  }
  __syncthreads();
  if (!s_walk) return;

  const int n1 = k, n2 = k * (k - 1) / 2, n3 = k * (k - 1) * (k - 2) / 6;
  const auto triple = [&](int u) {
    return u < n3 ? __ldg(g_tw_comb + tw_comb_off(3) + u) : 0u;
  };
  uint32_t next = triple(tid);
  for (int i = tid; i < n2; i += kTwPrepThreads) {
    if (i != tid) pair = __ldg(g_tw_comb + tw_comb_off(2) + i);
    const V6 &A = s_rows[pair & 31u], &Z = s_rows[pair >> 5];
    s_ratio[i].lo = tw_ratio(TwCols{A.l0, A.l1, A.l2}, TwCols{Z.l0, Z.l1, Z.l2});
    s_ratio[i].hi = tw_ratio(TwCols{A.h0, A.h1, A.h2}, TwCols{Z.h0, Z.h1, Z.h2});
  }
  __syncthreads();

  // Levels 1 to 3: seven sweeps per triple, one per pair, rows; the triples
  // first, so the short units even out the threads' loads.
  int wmin = kN + 1;
  for (int u = tid; u < n1 + n2 + n3; u += kTwPrepThreads) {
    if (u < n3) {
      const uint32_t rows = next, rz = rows >> 10;
      next = triple(u + kTwPrepThreads);  // on its way during the sweeps
      const TwRatio* by_z = s_ratio + rz * (rz - 1u) / 2u;
      const TwRatio &Q = by_z[rows & 31u], &X = by_z[(rows >> 5) & 31u];
      const uint32_t nz_lo = Q.lo.w, nz_hi = Q.hi.w;
      const TwCols lo = tw_cols(Q.lo), hi = tw_cols(Q.hi);
      TwCols x = tw_cols(X.lo), xh = tw_cols(X.hi);
#pragma unroll
      for (int s = 0; s < 7; ++s) {
        wmin = min(wmin, tw_least(tw_sum(lo, x), tw_sum(hi, xh), nz_lo, nz_hi));
        x = tw_alpha(x);
        xh = tw_alpha(xh);
      }
    } else if (u < n2 + n3) {
      const TwRatio& Q = s_ratio[u - n3];
      wmin = min(wmin, tw_least(tw_cols(Q.lo), tw_cols(Q.hi), Q.lo.w, Q.hi.w));
    } else {
      const V6& P = s_rows[u - n2 - n3];
      wmin = min(wmin, __popc(P.l0 | P.l1 | P.l2) + __popc(P.h0 | P.h1 | P.h2));
    }
  }
  const auto least = [&](int x) {
    x = __reduce_min_sync(0xffffffffu, x);
    __syncthreads();
    if (lane == 0) s_min[tid >> 5] = x;
    __syncthreads();
    for (int i = 0; i < kTwPrepThreads / 32; ++i) x = min(x, s_min[i]);
    return x;
  };
  wmin = least(wmin);
  int level = 3;
  bool p1 = false;
  unsigned long long words4 = 0ull;
  TwStage st{};
  if (k <= (a.n >= a.tw_ctas ? kTwPrepKBig : kTwPrepK)) {
    const int wthr = kN - a.desc[c].tmax;
    int l = level;
    bool p = p1;
    if (tw_next(k, wmin, wthr, l, p, st) && st.w == 4) {
      level = l;
      p1 = p;
      words4 = 343ull * c_binom[k - st.avoid() - st.forced()][4 - st.forced()];
      const int stop = tw_stop(k, st, wthr);
      wmin = least(k <= kTwWholeK ? tw_level4<true>(s_ratio, k, st, wmin, stop, tid)
                                  : tw_level4<false>(s_ratio, k, st, wmin, stop, tid));
    }
  }
  if (tid < 32) {
    if (lane == 0) {
      a.is_best[c] = wmin;
      atomicAdd(&a.is_hdr->codewords,
                static_cast<unsigned long long>(n1 + 7 * n2 + 49 * n3) + words4);
      if (words4) atomicAdd(&a.is_hdr->stage_codewords[st.forced() ? 8 : 9], words4);
    }
    __syncwarp();
    tw_advance(a, view, lane, c, k, level, p1, TwStage{}, 1u, true);
  }
}

// ---------------------------------------------------------------------------
// Walk
// ---------------------------------------------------------------------------

// A CTA's visit to a stage, prepared by warp 0.
struct TwJob {
  TwStage st;
  int c, k;
  unsigned int seq, claims;
  int stop;  // the code is decided at this weight or below
  int best;  // smallest weight met (this CTA's view)
  int last;  // no more work
  unsigned int first;          // the claim it came with
  unsigned int done;           // claims done in the visit
  unsigned long long words;    // codewords counted
  unsigned long long end[32];  // u's up to and with pivot row p
};

// Warp 0's view of the queue.
struct TwFetch {
  int c;       // the code worked on last (-1: none)
  bool waits;  // place `pos` of the queue is drawn, its ticket not yet seen
  bool drawn;  // the visit at hand came with a ticket
  unsigned int pos;
};

struct TwShared {
  TwJob job[2];            // the visit under way and the next one
  unsigned long long batch[kTwWarps];  // first u of the batch that a warp works on
  int held_c, held_block;  // whose bit rows are in the table
  TwFetch fetch;
};

__shared__ TwShared tw_s;
extern __shared__ __align__(1024) uint8_t tw_raw[];

// Calls f(row, exponent) for the rows of u number o of pivot row p.
template <typename F>
__device__ __forceinline__ void tw_for_rows(const TwStage& st, int k, int p, unsigned long long o,
                                            F f) {
  f(p, 0u);
  const int picks = st.w - 3 - st.forced();
  if (st.forced()) {
    const unsigned long long q = o / 7u;
    f(k - 1, static_cast<uint32_t>(o - 7u * q));
    o = q;
  }
  uint32_t dig = 0u;  // picks <= 8
  if (o >> 32) {
    for (int j = 0; j < picks; ++j) {
      const unsigned long long q = o / 7u;
      dig |= static_cast<uint32_t>(o - 7u * q) << (3 * j);
      o = q;
    }
  } else {
    uint32_t x = static_cast<uint32_t>(o);
    for (int j = 0; j < picks; ++j) {
      const uint32_t q = x / 7u;
      dig |= (x - 7u * q) << (3 * j);
      x = q;
    }
    o = x;
  }
  if (picks <= 4) {
    uint32_t rows = picks ? __ldg(g_tw_comb + tw_comb_off(picks) + static_cast<uint32_t>(o)) : 0u;
    for (int j = 0; j < picks; ++j) {
      f(p + 1 + int(rows & 31u), dig & 7u);
      rows >>= 5;
      dig >>= 3;
    }
  } else {
    int r = k;
    for (int j = picks; j > 0; --j) {
      do --r;
      while (c_binom[r][j] > o);
      o -= c_binom[r][j];
      f(p + 1 + r, dig & 7u);
      dig >>= 3;
    }
  }
}

// Rows and exponents of pair e.
struct TwPair {
  uint32_t lo, hi, d_lo, d_hi;
};

__device__ __forceinline__ TwPair tw_pair(uint32_t e) {
  const uint32_t pick = e / 49u, d = e - 49u * pick;
  const uint32_t rows = __ldg(g_tw_comb + 21 + pick);
  return TwPair{rows & 31u, rows >> 5, d / 7u, d % 7u};
}

// Weight, over all 49 columns, of u number o of pivot row p plus pair e.
__device__ __forceinline__ int tw_weight(const V6* rows, const TwStage& st, int k, int p,
                                         unsigned long long o, uint32_t e) {
  V6 P;
  v6_zero(P);
  const auto add = [&](int r, uint32_t x) {
    V6 g = v6_ldg(rows + r);
    v6_alpha_pow(g, int(x));
    v6_xor(P, g);
  };
  tw_for_rows(st, k, p, o, add);
  const TwPair q = tw_pair(e);
  add(int(q.lo), q.d_lo);
  add(int(q.hi), q.d_hi);
  return __popc(lop3<0xFE>(P.l0, P.l1, P.l2)) + __popc(lop3<0xFE>(P.h0, P.h1, P.h2));
}

// Transposes a 32 x 32 bit matrix, row i in lane i.
__device__ __forceinline__ uint32_t tw_transpose(uint32_t x, int lane) {
  uint32_t mask = 0x0000FFFFu;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, s);
    const bool up = (lane & s) != 0;
    const uint32_t r = __funnelshift_l(y, y, up ? 32 - s : s);
    const uint32_t keep = up ? ~mask : mask;
    x = lop3<0xCA>(keep, x, r);  // keep ? x : r
    mask ^= mask << (s >> 1);
  }
  return x;
}

// The words of the eight values in four 32-pair words of a column, given as
// three planes each.
__device__ __forceinline__ void tw_put(uint8_t* dst, const uint32_t (&t)[4][3]) {
#pragma unroll
  for (int val = 0; val < 8; ++val) {
    uint32_t z[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      z[q] = (val & 1 ? t[q][0] : ~t[q][0]) & (val & 2 ? t[q][1] : ~t[q][1]) &
             (val & 4 ? t[q][2] : ~t[q][2]);
    *reinterpret_cast<uint4*>(dst + 16 * val) = make_uint4(z[0], z[1], z[2], z[3]);
  }
}

// The bit rows of the code's pairs from the block's first on: a warp takes four
// words, computes a pair's values per lane, transposes the planes (lane:
// column) and writes the eight values' words.
template <typename L>
__device__ __forceinline__ void tw_build(const uint4* tab, int k, int block, int warp, int lane) {
  const uint32_t all = 49u * static_cast<uint32_t>(c_binom[k - 2][2]);
  const uint32_t first = static_cast<uint32_t>(block) * L::kPairs;
  const uint32_t words = min((all - first + 31u) / 32u, static_cast<uint32_t>(L::kWords));
  for (uint32_t g = warp; 4u * g < words; g += kTwWarps) {
    uint32_t t[4][3], ext[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const TwPair e = tw_pair(min(first + 128u * g + 32u * q + lane, all - 1u));
      const uint4 x = __ldg(tab + e.lo * 7u + e.d_lo), y = __ldg(tab + e.hi * 7u + e.d_hi);
      t[q][0] = tw_transpose(x.x ^ y.x, lane);
      t[q][1] = tw_transpose(x.y ^ y.y, lane);
      t[q][2] = tw_transpose(x.z ^ y.z, lane);
      if (L::kCols > 32) ext[q] = tw_transpose(x.w ^ y.w, lane);
    }
    uint8_t* dst = tw_raw + lane * L::kColBytes + g * 128u;
    tw_put(dst, t);
    if (L::kCols > 32) {
      // planes of column 32 + l: lanes l, 10 + l, 20 + l
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        t[q][0] = ext[q];
        t[q][1] = __shfl_sync(0xffffffffu, ext[q], lane + 10);
        t[q][2] = __shfl_sync(0xffffffffu, ext[q], lane + 20);
      }
      if (lane < L::kCols - 32) tw_put(dst + 32 * L::kColBytes, t);
      __syncwarp();
    }
  }
}

// alpha^e g of every row as one byte per column, 16 times the value: the
// offset of the value's words in a column's group.
template <typename L>
__device__ __forceinline__ void tw_spread_rows(const uint4* tab, int k, int tid) {
  for (int i = tid; i < 7 * k; i += kTwThreads) {
    const uint4 x = __ldg(tab + i);
    uint32_t* dst = reinterpret_cast<uint32_t*>(tw_raw + L::kTableBytes + i * L::kRowBytes);
    const auto put = [&](int j, uint32_t p0, uint32_t p1, uint32_t p2) {
      const auto bits = [](uint32_t four) { return ((four & 15u) * 0x00204081u) & 0x01010101u; };
      dst[j] = (bits(p0) << 4) | (bits(p1) << 5) | (bits(p2) << 6);
    };
#pragma unroll
    for (int j = 0; j < 8; ++j) put(j, x.x >> (4 * j), x.y >> (4 * j), x.z >> (4 * j));
    if (L::kCols > 32) {
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const uint32_t m = j < 2 ? 15u : 3u;  // ten columns
        put(8 + j, (x.w >> (4 * j)) & m, (x.w >> (10 + 4 * j)) & m, (x.w >> (20 + 4 * j)) & m);
      }
      dst[11] = 0u;
    }
  }
}

// Full adder on four words: s, a, b -> sum in s; returns the carries.
struct TwW4 {
  uint32_t x[4];
};

__device__ __forceinline__ TwW4 tw_add(TwW4& s, const TwW4& a, const TwW4& b) {
  TwW4 c;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    c.x[i] = lop3<0xE8>(s.x[i], a.x[i], b.x[i]);
    s.x[i] = lop3<0x96>(s.x[i], a.x[i], b.x[i]);
  }
  return c;
}

__device__ __forceinline__ TwW4 tw_splat(uint32_t x) { return TwW4{{x, x, x, x}}; }

// For the 128 pairs of a group, whose offset is `at` (a multiple of 256) plus
// bit 7 of u's bytes: bit set where u plus the pair has at least kTop - bias zeros among
// the first C columns, kTop = 32 or 64.  u: the lane's value offsets, a byte
// per column.
template <typename L, int C>
__device__ __forceinline__ TwW4 tw_count(const uint32_t (&u)[L::kRowBytes / 4], uint32_t at,
                                         uint32_t bias) {
  const auto row = [&](int col) {
    // the column's byte becomes the offset's low byte
    const uint32_t o = __byte_perm(u[col >> 2], at, 0x7650 | (col & 3));
    const uint4 x = *reinterpret_cast<const uint4*>(tw_raw + col * L::kColBytes + o);
    return TwW4{{x.x, x.y, x.z, x.w}};
  };
  const auto bit = [&](int i) { return tw_splat(0u - ((bias >> i) & 1u)); };
  static_assert(C % 2 == 0 && C <= L::kCols, "columns");
  constexpr int kLevels = C <= 32 ? 5 : 6;
  // counters of weight 1, 2, 4, ..., started at the bias, and for each weight
  // a row that waits for a second one
  TwW4 n[kLevels], wait[kLevels + 1];
#pragma unroll
  for (int l = 0; l < kLevels; ++l) n[l] = bit(l);
#pragma unroll
  for (int i = 0; i < C / 2; ++i) {
    TwW4 carry = tw_add(n[0], row(2 * i), row(2 * i + 1));
#pragma unroll
    for (int l = 1; l <= kLevels; ++l) {
      if (l == kLevels || !((i >> (l - 1)) & 1)) {
        wait[l] = carry;
        break;
      }
      carry = tw_add(n[l], wait[l], carry);
    }
  }
  // what waits is counted from the lowest weight up; the carry out of the
  // highest counter is the result
  TwW4 over{}, carry{};
  bool have = false, out = false;
#pragma unroll
  for (int l = 1; l < kLevels; ++l) {
    const bool waits = ((C / 2) >> (l - 1)) & 1;
    if (!waits && !have) continue;
    carry = tw_add(n[l], waits ? wait[l] : tw_splat(0u), have ? carry : tw_splat(0u));
    have = true;
  }
  if ((C / 2) >> (kLevels - 1)) {
    over = wait[kLevels];
    out = true;
  }
  if (!have) return over;
#pragma unroll
  for (int i = 0; i < 4; ++i) over.x[i] = out ? over.x[i] | carry.x[i] : carry.x[i];
  return over;
}

// A lane's u: the x-th of the stage, counted from the last pivot row's down (the
// longest lists first).
struct TwU {
  int p;
  unsigned long long o;  // its number among those of pivot row p
  uint32_t nv;           // pairs below p
};

__device__ __forceinline__ TwU tw_u(const TwJob& J, unsigned long long x) {
  const unsigned long long total = J.end[31];
  x = total - 1ull - min(x, total - 1ull);
  int p = 0;  // pivot rows with end <= x
#pragma unroll
  for (int s = 16; s > 0; s >>= 1)
    if (J.end[p + s - 1] <= x) p += s;
  return TwU{p, x - (p ? J.end[p - 1] : 0ull), tw_pairs_below(p)};
}

// Weighs the pairs of the block from e0 on that passed for this lane's u.
__device__ __forceinline__ void tw_light(const DistArgs& a, TwJob& J, unsigned long long batch,
                                         const TwW4& hit, uint32_t all, uint32_t e0) {
  const TwStage st = J.st;
  const TwU u = tw_u(J, batch + (threadIdx.x & 31u));
  const uint32_t first = static_cast<uint32_t>(st.block) * tw_pairs(J.k) + e0;
  const V6* rows = tw_view(a).rows + size_t(J.c) * a.k_max;
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    uint32_t m = (q == 0 ? hit.x[0] : q == 1 ? hit.x[1] : q == 2 ? hit.x[2] : hit.x[3]) | all;
    for (; m != 0u; m &= m - 1u) {
      const uint32_t e = first + 32u * q + (__ffs(int(m)) - 1);
      if (e >= u.nv) break;
      const int wt = tw_weight(rows, st, J.k, u.p, u.o, e);
      if (wt < *reinterpret_cast<volatile int*>(&J.best)) {
        atomicMin(&J.best, wt);
        atomicMin(a.is_best + J.c, wt);
      }
    }
  }
}

// One piece of a batch: 32 u's (one per lane) against pairs begin..end of the
// block.  Pairs that a lane's u does not have are left to tw_light.
template <typename L, int C>
__device__ __forceinline__ void tw_batch(const DistArgs& a, TwJob& J,
                                         const unsigned long long& batch,
                                         uint32_t (&u)[L::kRowBytes / 4], uint32_t begin,
                                         uint32_t end, int allowed) {
  constexpr int kTop = C <= 32 ? 32 : 64;
  const int need = C - allowed;  // zeros among the C columns
  const uint32_t all = need <= 0 ? ~0u : 0u;
  const uint32_t bias = need <= 0 ? 0u : static_cast<uint32_t>(kTop - need);
#pragma unroll 1
  for (uint32_t e0 = begin; e0 < end; e0 += 128u) {
    const TwW4 hit = tw_count<L, C>(u, e0 & ~255u, bias);
#pragma unroll
    for (int i = 0; i < L::kRowBytes / 4; ++i) u[i] ^= 0x80808080u;
    if (lop3<0xFE>(hit.x[0], hit.x[1], hit.x[2]) | hit.x[3] | all)  // rare
      tw_light(a, J, batch, hit, all, e0);
  }
}

// A warp's share of the CTA's visit: claims, one at a time, the next one on its
// way while it works.
template <typename L>
__device__ __forceinline__ void tw_walk(const DistArgs& a, const TwView& v, TwJob& J, int warp,
                                        int lane) {
  const TwStage st = J.st;
  const int k = J.k;
  const unsigned long long n_u = J.end[31], total = (n_u + 31ull) / 32ull << st.cut;
  const unsigned int claims = J.claims, seq = J.seq;
  unsigned long long* counter = &v.state[J.c].claim;
  unsigned long long words = 0ull, next = 0ull;
  unsigned int done = 0u;
  if (lane == 0)
    next = warp == 0 ? (static_cast<unsigned long long>(seq) << 32) | J.first
                     : atomicAdd(counter, 1ull);
  for (;;) {
    const unsigned long long cl = __shfl_sync(0xffffffffu, next, 0);
    if (static_cast<unsigned int>(cl >> 32) != seq || static_cast<unsigned int>(cl) >= claims)
      break;
    ++done;
    const int best = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile int*>(&J.best), 0);
    if (best <= J.stop) {
      // decided: what nobody has claimed is skipped at once
      unsigned long long old = 0ull;
      if (lane == 0)
        old = atomicMax(counter, (static_cast<unsigned long long>(seq) << 32) | claims);
      old = __shfl_sync(0xffffffffu, old, 0);
      if (static_cast<unsigned int>(old) < claims) done += claims - static_cast<unsigned int>(old);
      break;
    }
    if (lane == 0) {
      next = atomicAdd(counter, 1ull);
      if ((done & 15u) == 0u) atomicAdd(&v.hdr->progress, 1u);
    }
    for (unsigned long long i = static_cast<unsigned int>(cl); i < total; i += claims) {
      const unsigned long long batch = i >> st.cut;
      const uint32_t piece = static_cast<uint32_t>(i - (batch << st.cut));
      if (lane == 0) tw_s.batch[warp] = 32ull * batch;
      const TwU x = tw_u(J, 32ull * batch + lane);
      const uint32_t nv = min(x.nv - static_cast<uint32_t>(st.block) * L::kPairs,
                              static_cast<uint32_t>(L::kPairs));
      // the piece's groups of 128 pairs
      const uint32_t groups = (__reduce_max_sync(0xffffffffu, nv) + 127u) / 128u;
      const uint32_t per = (groups + (1u << st.cut) - 1u) >> st.cut;
      const uint32_t begin = 128u * piece * per;
      const uint32_t end = 128u * min(groups, (piece + 1u) * per);
      if (begin >= end) continue;
      if (32ull * batch + lane < n_u && nv > begin) words += min(nv, end) - begin;
      uint32_t u[L::kRowBytes / 4];
#pragma unroll
      for (int q = 0; q < L::kRowBytes / 4; ++q) u[q] = begin & 128u ? 0x80808080u : 0u;
      tw_for_rows(st, k, x.p, x.o, [&](int r, uint32_t e) {
        const uint4* src =
            reinterpret_cast<const uint4*>(tw_raw + L::kTableBytes + (r * 7u + e) * L::kRowBytes);
#pragma unroll
        for (int q = 0; q < L::kRowBytes / 16; ++q) {
          const uint4 y = src[q];
          u[4 * q] ^= y.x;
          u[4 * q + 1] ^= y.y;
          u[4 * q + 2] ^= y.z;
          u[4 * q + 3] ^= y.w;
        }
      });
      __syncwarp();
      // The fewest columns that let less than about 1e-6 of random codewords
      // pass (weighing one holds up its warp for two thousand cycles): 15 zeros
      // of 30, 16 of 36; 42 are all columns of k >= 7.  (At k = 20 and 21, 29
      // and 28 columns lie outside E; the others are zero in every row.)
      const int allowed = best - 1 - st.w;
      const unsigned long long& b = tw_s.batch[warp];
      if constexpr (L::kCols == 32) {
        if (allowed <= 15) tw_batch<L, 30>(a, J, b, u, begin, end, allowed);
        else tw_batch<L, 32>(a, J, b, u, begin, end, allowed);
      } else {
        if (allowed <= 20) tw_batch<L, 36>(a, J, b, u, begin, end, allowed);
        else tw_batch<L, 42>(a, J, b, u, begin, end, allowed);
      }
      __syncwarp();
    }
  }
  for (int o = 16; o > 0; o >>= 1) words += __shfl_xor_sync(0xffffffffu, words, o);
  if (lane == 0) {
    if (words) atomicAdd(&J.words, words);
    if (done) atomicAdd(&J.done, done);
  }
}

// Counts what the CTA has done in a visit (warp 0); whoever counts a stage's
// last claim settles the code or opens its next stage.
__device__ __noinline__ void tw_finish(const DistArgs& a, int lane, int job) {
  const TwView v = tw_view(a);
  const TwJob& J = tw_s.job[job];
  if (lane == 0 && J.words) {
    atomicAdd(&a.is_hdr->codewords, J.words);
    atomicAdd(&a.is_hdr->stage_codewords[2 * J.st.w + (J.st.forced() ? 0 : 1)], J.words);
  }
  unsigned int n = 0u;
  if (lane == 0) {
    __threadfence();
    n = atomicAdd(&v.state[J.c].done, J.done) + J.done;
    __threadfence();
    atomicAdd(&v.hdr->progress, 1u);
  }
  n = __shfl_sync(0xffffffffu, n, 0);
  if (n != J.claims) return;
  const volatile TwState& s = v.state[J.c];
  const int level = s.level;
  __syncwarp();
  tw_advance(a, v, lane, J.c, J.k, level & 63, (level & 64) != 0, J.st, J.seq + 1u, false);
}

__device__ __forceinline__ uint4 tw_ld_acquire4(const void* p) {
  uint4 v;
  asm volatile("ld.acquire.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

// Looks at code c's stage and prepares a visit to it: the stage of the claim
// `held` (stage number << 32 | claim), or, where that is 0, the one under way.
// False when there is nothing to claim.
__device__ __forceinline__ bool tw_look(const DistArgs& a, const TwView& v, int lane, int c,
                                        unsigned long long held, TwJob& J) {
  const int k = a.desc[c].k, tmax = a.desc[c].tmax, best = ld_flag(a.is_best + c);
  unsigned int seq = 0u, claims = 0u, w = 0u;
  if (lane == 0) {
    const uint4 x = tw_ld_acquire4(&v.state[c].claim);
    const uint4 y = tw_ld_acquire4(&v.state[c].seq);
    const unsigned int next = held ? static_cast<unsigned int>(held) : x.x;
    seq = held ? static_cast<unsigned int>(held >> 32) : x.y;
    // a stage that is being replaced has its number changed first
    if (x.y == seq && y.x == seq && next < x.z) claims = x.z;
    w = y.y;
  }
  claims = __shfl_sync(0xffffffffu, claims, 0);
  if (claims == 0u) return false;
  w = __shfl_sync(0xffffffffu, w, 0);
  const TwStage st{int8_t(w), int8_t(w >> 8), int8_t(w >> 16), int8_t(w >> 24)};
  unsigned long long words = 0ull;
  const unsigned long long end = tw_ends(k, st, lane, words);
  J.end[lane] = end;
  if (lane == 0) {
    J.st = st;
    J.c = c;
    J.k = k;
    J.seq = seq;
    J.claims = claims;
    J.stop = tw_stop(k, st, kN - tmax);
    J.best = best;
    J.last = 0;
    J.done = 0u;
    J.words = 0ull;
  }
  __syncwarp();
  return true;
}

// Takes the first claim of the visit; false when none is left.  (Not by
// comparing: under the other warps' claims that never succeeds.)  Where the
// code's next stage has begun meanwhile, the claim is one of that stage, and
// the visit goes there.  Later claims of the visit are of its stage, which
// cannot end before this one is counted.
__device__ __forceinline__ bool tw_claim(const DistArgs& a, const TwView& v, int lane, TwJob& J) {
  unsigned long long cl = 0ull;
  if (lane == 0) cl = atomicAdd(&v.state[J.c].claim, 1ull);
  cl = __shfl_sync(0xffffffffu, cl, 0);
  if (static_cast<unsigned int>(cl >> 32) != J.seq) {
    const int c = J.c;
    __syncwarp();
    if (!tw_look(a, v, lane, c, cl, J)) return false;
  }
  if (lane == 0) J.first = static_cast<unsigned int>(cl);
  __syncwarp();
  return static_cast<unsigned int>(cl) < J.claims;
}

// Takes the ticket at the drawn place, if it is there (one thread): the code
// plus one, or 0.
__device__ __forceinline__ unsigned int tw_ticket(const TwView& v, unsigned int pos) {
  unsigned int* slot = v.queue + pos % v.cap;
  const unsigned int entry = tw_ld_acquire(slot);
  if (entry == 0u || entry == kTwOver) return entry;
  tw_st_release(slot, 0u);
  atomicSub(&v.state[entry - 1u].tickets, 1);
  __threadfence();  // before the look at its stage
  return entry;
}

// The visit in J came with a ticket: others may join in, those that wait now
// and one later, while twice as many claims are left as a CTA's warps take at
// once.  (One at a time, a lone code's last CTA would join a millisecond after
// the first.)
__device__ __forceinline__ void tw_pass_on(const DistArgs& a, const TwView& v, int lane,
                                           const TwJob& J) {
  const unsigned int first = J.first;
  if (first + 2u * kTwWarps > J.claims) return;
  tw_push(a, v, lane, J.c,
          min(max(tw_waiting(v), 1), int((J.claims - first) / (2u * kTwWarps))));
}

// The CTA's next visit, claim included: to the code at hand while its stage has
// claims, else to the queue's next code.  False when no code is open any more.
__device__ __noinline__ bool tw_fetch(const DistArgs& a, int lane, int job) {
  const TwView v = tw_view(a);
  TwJob& J = tw_s.job[job];
  TwFetch& f = tw_s.fetch;
  int c = f.c;
  bool drawn = false;
  for (;;) {
    if (c >= 0 && tw_look(a, v, lane, c, 0ull, J) && tw_claim(a, v, lane, J)) {
      if (lane == 0) {
        f.c = c;
        f.drawn = drawn;
      }
      __syncwarp();
      return true;
    }
    unsigned int entry = kTwOver;
    if (lane == 0 && *reinterpret_cast<volatile int*>(&v.hdr->open) != 0) {
      if (!f.waits) f.pos = atomicAdd(&v.hdr->head, 1u);
      f.waits = false;
      unsigned int seen = 0u;
      // Only this CTA looks at its place in the queue: with a common word
      // watched by all, the one that opens a stage waited for them (70 us).
      // 2^22 looks of 0.1 us and more without work ending anywhere: give up.
      for (unsigned int i = 0; i < (1u << 22); ++i) {
        entry = tw_ticket(v, f.pos);
        if (entry != 0u) break;
        if ((i & 1023u) == 1023u) {
          const unsigned int pr = *reinterpret_cast<volatile unsigned int*>(&v.hdr->progress);
          if (pr != seen) {
            seen = pr;
            i = 0;
          }
        }
        if (i + 1 == (1u << 22)) {
          report_status(a.hdr, TG_ERR_TIMEOUT);
          entry = kTwOver;
        }
        __nanosleep(100);
      }
    }
    entry = __shfl_sync(0xffffffffu, entry, 0);
    if (entry == kTwOver) return false;
    c = int(entry) - 1;
    drawn = true;
  }
}

// Prepares the next visit, without a claim, while the other warps work: a dozen
// round trips to L2 that nobody waits for.  Only while the queue holds a ticket
// for every CTA; at its end a code goes to whoever is idle.
__device__ __noinline__ bool tw_prefetch(const DistArgs& a, int lane, int job) {
  const TwView v = tw_view(a);
  TwJob& J = tw_s.job[job];
  TwFetch& f = tw_s.fetch;
  for (;;) {
    unsigned int entry = 0u;
    if (lane == 0) {
      if (!f.waits) {
        const unsigned int head = *reinterpret_cast<volatile unsigned int*>(&v.hdr->head);
        const unsigned int tail = *reinterpret_cast<volatile unsigned int*>(&v.hdr->tail);
        if (int(tail - head) > a.tw_ctas) {
          f.pos = atomicAdd(&v.hdr->head, 1u);
          f.waits = true;
        }
      }
      if (f.waits) entry = tw_ticket(v, f.pos);
      if (entry == kTwOver) entry = 0u;
      if (entry) f.waits = false;
    }
    entry = __shfl_sync(0xffffffffu, entry, 0);
    __syncwarp();
    if (entry == 0u) return false;
    const int c = int(entry) - 1;
    if (tw_look(a, v, lane, c, 0ull, J)) {
      if (lane == 0) {
        f.c = c;
        f.drawn = true;
      }
      __syncwarp();
      return true;
    }
  }
}

// What warp 0 does while the other warps begin a visit: it lets others join,
// counts the visit before and looks for the next one.
__device__ __noinline__ bool tw_duties(const DistArgs& a, int lane, int cur, bool pending) {
  if (tw_s.fetch.drawn) tw_pass_on(a, tw_view(a), lane, tw_s.job[cur]);
  __syncwarp();
  if (lane == 0) tw_s.fetch.drawn = false;
  __syncwarp();
  if (pending) tw_finish(a, lane, cur ^ 1);
  return tw_prefetch(a, lane, cur ^ 1);
}

__global__ void __launch_bounds__(kTwThreads, kTwCtasPerSm) toric_walk_kernel(
    const __grid_constant__ DistArgs a) {
  const TwView v = tw_view(a);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    tw_s.held_c = -1;
    tw_s.held_block = 0;
    tw_s.fetch.c = -1;
    tw_s.fetch.waits = tw_s.fetch.drawn = false;
  }
  __syncwarp();
  if (warp == 0 && !tw_fetch(a, lane, 0) && lane == 0) tw_s.job[0].last = 1;
  bool pending = false;  // (warp 0) the visit before is not counted yet
  for (int cur = 0;; cur ^= 1) {
    __syncthreads();
    TwJob& J = tw_s.job[cur];
    if (J.last) return;
    if (tw_s.held_c != J.c || tw_s.held_block != J.st.block) {
      const uint4* tab = v.tab + size_t(J.c) * a.k_max * 7;
      if (J.k <= kTwWideK) {
        tw_spread_rows<TwWide>(tab, J.k, tid);
        tw_build<TwWide>(tab, J.k, J.st.block, warp, lane);
      } else {
        tw_spread_rows<TwNarrow>(tab, J.k, tid);
        tw_build<TwNarrow>(tab, J.k, J.st.block, warp, lane);
      }
      __syncthreads();
      if (tid == 0) {
        tw_s.held_c = J.c;
        tw_s.held_block = J.st.block;
      }
    }
    bool more = false;
    if (warp == 0) more = tw_duties(a, lane, cur, pending);
    if (J.k <= kTwWideK) tw_walk<TwWide>(a, v, J, warp, lane);
    else tw_walk<TwNarrow>(a, v, J, warp, lane);
    __threadfence();  // is_best before the visit is counted
    __syncthreads();
    if (warp == 0) {
      pending = more && tw_claim(a, v, lane, tw_s.job[cur ^ 1]);
      if (!pending) {
        // nothing at hand: this visit may be what the next one waits for
        if (lane == 0) tw_s.fetch.drawn = false;
        tw_finish(a, lane, cur);
        if (!tw_fetch(a, lane, cur ^ 1) && lane == 0) tw_s.job[cur ^ 1].last = 1;
      }
    }
  }
}

// Per-device tables and launch attributes (with the device current).
int tw_upload_tables() {
  std::vector<uint32_t> comb;
  for (int b = 1; b <= 4; ++b) {
    int r[4];
    for (int i = 0; i < b; ++i) r[i] = i;
    for (;;) {
      uint32_t x = 0;
      for (int i = 0; i < b; ++i) x |= uint32_t(r[i]) << (5 * i);
      comb.push_back(x);
      int i = 0;
      while (i < b && r[i] + 1 == (i + 1 < b ? r[i + 1] : kMaxExactK)) ++i;
      if (i == b) break;
      ++r[i];
      for (int j = 0; j < i; ++j) r[j] = j;
    }
  }
  cudaError_t e = cudaMemcpyToSymbol(g_tw_comb, comb.data(), comb.size() * sizeof(uint32_t));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(toric_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kTwSharedBytes);
  return e == cudaSuccess ? TG_OK : cuda_fail(e, "toric walk tables");
}

}  // namespace tg
