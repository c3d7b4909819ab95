// Sampled screening (kernel_cuda_bp.py:167-236): work ids 1..sample_count, the
// message from a splitmix64 hash of (seed, set id, work id), bit-exact to the
// reference.  Included by distance.cu, whose tables, descriptors and helpers
// it shares.
//
// A message is 3 k bits, and the codeword is the GF(2) sum of the vectors of
// the bits that are set.  A CTA lays out, for each five consecutive bits, the
// 32 sums of their vectors in shared memory, packed into five words (planes of
// columns 0..31, then those of columns 32..41 and of 42..48 in one word each),
// every word's 32 entries in a row of their own: a lane's five bits select its
// bank, so 32 lanes with 32 different messages read a word without conflicts.
// Five bits are the most that do (a quarter of the lookups by eight-entry
// tables of 16-byte words would be: 3 bits a cycle of the shared-memory pipe,
// here 5).  For 3 k <= 63 one hash gives all bits and the lookups bound the
// kernel; above that each coefficient has its own hash, and its 14 logic and
// 6 multiply instructions do (about 7 cycles per coefficient, warp and SM,
// against 3 of the lookups).  2,000 sets of 16..30 rows, 3,000 samples each:
// kernel 0.20 ms, Python call 0.91 -> 0.42 ms (before, a lane added k vectors
// of 32 bytes through L1 for each sample, 64 samples in a row).
#pragma once

namespace tg {

constexpr uint64_t kSampleChunk = 64;  // work ids per counted task
constexpr int kScreenThreads = 128;
constexpr int kScreenGroupWords = 5 * 32;

// Five-bit groups of a k-row table: whole chunks of five rows (three groups),
// and one more, so that groups can be taken in pairs.
__host__ __device__ constexpr int screen_groups(int k) { return (k + 4) / 5 * 3 + 1; }

__host__ __device__ constexpr int screen_shared_bytes(int k_max) {
  return (screen_groups(k_max) * kScreenGroupWords + k_max * 3 * 5) * 4;
}

__global__ void __launch_bounds__(kPrepWarps * 32) prep_sampled_kernel(DistArgs a) {
  const int w = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * kPrepWarps + w;
  if (c >= a.n) return;
  const int64_t beg = a.off[c];
  const int64_t klong = a.off[c + 1] - beg;
  const bool ok_k = klong >= 0 && klong <= a.k_max;
  const int k = ok_k ? int(klong) : 0;
  bool bad = !ok_k;
  V6* rows = a.bitpat + size_t(c) * a.bitpat_stride;
  for (int i = lane; i < k; i += 32) {  // k <= 49
    const int r = a.idx[beg + i];
    if (r < 0 || r >= kN) {
      bad = true;
      continue;
    }
    const uint64_t* p = a.tab.Mp + r * 3;
    v6_stg(rows + i, v6_of_planes(__ldg(p), __ldg(p + 1), __ldg(p + 2)));
  }
  bad = __any_sync(0xffffffffu, bad);
  if (lane != 0) return;
  if (bad) report_status(a.hdr, TG_ERR_BAD_INPUT);
  CodeDesc d{};
  d.k = k;
  d.set_id = a.set_ids ? a.set_ids[c] : c;
  d.tmax = kN - (a.target ? a.target[c] : a.td_default);
  d.n_tasks = bad || k == 0 ? 0ull : (uint64_t(a.sample_count) + kSampleChunk - 1) / kSampleChunk;
  a.desc[c] = d;
  // the reference evaluates the empty message sum, the zero codeword
  a.out[c] = !bad && k == 0 ? kN : 0;
  a.abort[c] = 0;
  if (d.n_tasks) {
    atomicAdd(&a.hdr->codewords, static_cast<unsigned long long>(a.sample_count));
    const unsigned long long old = atomicAdd(&a.hdr->total_tasks, d.n_tasks);
    if (old + d.n_tasks < old) {  // more than 2^64 tasks: nothing runs
      report_status(a.hdr, TG_ERR_INVALID_ARGUMENT);
      a.hdr->has_tasks = -1;
    }
  }
}

// A bit-sliced vector as five words.
__device__ __forceinline__ void screen_pack(const V6& g, uint32_t (&x)[5]) {
  x[0] = g.l0;
  x[1] = g.l1;
  x[2] = g.l2;
  x[3] = (g.h0 & 0x3FFu) | ((g.h1 & 0x3FFu) << 10) | ((g.h2 & 0x3FFu) << 20);
  x[4] = (g.h0 >> 10) | ((g.h1 >> 10) << 7) | ((g.h2 >> 10) << 14);
}

__device__ __forceinline__ int screen_weight(const uint32_t (&x)[5]) {
  const uint32_t ten = lop3<0xFE>(x[3], x[3] >> 10, x[3] >> 20) & 0x3FFu;
  const uint32_t seven = lop3<0xFE>(x[4], x[4] >> 7, x[4] >> 14) & 0x7Fu;
  return __popc(lop3<0xFE>(x[0], x[1], x[2])) + __popc(ten | (seven << 10));
}

// x + the group's entries e and the next group's f.
__device__ __forceinline__ void screen_add2(uint32_t (&x)[5], const uint32_t* group, uint32_t e,
                                            uint32_t f) {
#pragma unroll
  for (int w = 0; w < 5; ++w)
    x[w] = lop3<0x96>(x[w], group[32 * w + e], group[kScreenGroupWords + 32 * w + f]);
}

__device__ __forceinline__ void screen_add(uint32_t (&x)[5], const uint32_t* group, uint32_t e) {
#pragma unroll
  for (int w = 0; w < 5; ++w) x[w] ^= group[32 * w + e];
}

// x mod k for k <= 49, with inv = floor(2^32 / k) and r32 = 2^32 mod k.
__device__ __forceinline__ uint32_t screen_mod(uint64_t x, uint32_t k, uint32_t inv, uint32_t r32) {
  const auto mod = [&](uint32_t y) {
    const uint32_t r = y - __umulhi(y, inv) * k;  // < 2 k: the quotient is at most 1 too small
    return min(r, r - k);
  };
  return mod(mod(uint32_t(x >> 32)) * r32 + mod(uint32_t(x)));
}

// CTA b: work ids of piece b / n of code b % n, `passes` rounds of one per
// thread (so a code that fails its threshold does so in an early CTA).
__global__ void __launch_bounds__(kScreenThreads) screen_kernel(DistArgs a, uint64_t passes) {
  extern __shared__ uint32_t screen_raw[];
  const int c = blockIdx.x % a.n;
  const uint64_t piece = blockIdx.x / a.n;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const CodeDesc d = a.desc[c];
  if (d.n_tasks == 0 || a.hdr->has_tasks < 0) return;
  const int k = d.k, groups = screen_groups(k);
  uint32_t* table = screen_raw;
  uint32_t* vec = screen_raw + groups * kScreenGroupWords;  // five words per bit
  if (tid < k) {
    V6 g = v6_ldg(a.bitpat + size_t(c) * a.bitpat_stride + tid);
    for (int b = 0; b < 3; ++b) {
      uint32_t x[5];
      screen_pack(g, x);
      for (int w = 0; w < 5; ++w) vec[(3 * tid + b) * 5 + w] = x[w];
      v6_alpha_pow(g, 1);
    }
  }
  // Another CTA of the code may set the flag meanwhile: one thread looks at it
  // for all, since the table below is laid out by every warp or not at all.
  if (__syncthreads_or(tid == 0 && ld_flag(a.abort + c))) return;
  for (int g = warp; g < groups; g += kScreenThreads / 32) {
    uint32_t x[5] = {0u, 0u, 0u, 0u, 0u};
    for (int b = 0; b < 5 && 5 * g + b < 3 * k; ++b) {
      const uint32_t on = 0u - ((uint32_t(lane) >> b) & 1u);
      for (int w = 0; w < 5; ++w) x[w] ^= vec[(5 * g + b) * 5 + w] & on;
    }
    for (int w = 0; w < 5; ++w) table[g * kScreenGroupWords + 32 * w + lane] = x[w];
  }
  __syncthreads();

  constexpr uint64_t kRowStep = 0x94D049BB133111EBull;
  const uint64_t count = uint64_t(a.sample_count);
  const uint64_t first = piece * passes * kScreenThreads;  // work ids less one
  const uint64_t end = min(count, first + passes * kScreenThreads);
  const uint64_t seed_row = a.seed ^ (uint64_t(int64_t(d.set_id)) * 0x9E3779B97F4A7C15ull);
  const uint64_t seed_forced = a.seed ^ (uint64_t(int64_t(d.set_id)) * 0xD6E8FEB86659FD93ull);
  const bool poly = 3 * k <= 63;
  const uint32_t uk = uint32_t(k), r32 = uint32_t((1ull << 32) % uk);
  const uint32_t inv = poly ? 0u : uint32_t((1ull << 32) / uk);
  const int wthr = kN - d.tmax;  // abort when a weight < wthr appears
  int wmin = kN;
  for (uint64_t at = first; at < end; at += kScreenThreads) {
    const int stop = ld_flag(a.abort + c);
    const uint64_t wid = min(at + uint64_t(tid), end - 1) + 1ull;  // past the end: the last again
    const uint64_t base = seed_row ^ (wid * 0xBF58476D1CE4E5B9ull);
    uint32_t x[5] = {0u, 0u, 0u, 0u, 0u};
    if (poly) {
      const uint64_t pid = mod_mersenne(splitmix64(base), 3 * k) + 1ull;
#pragma unroll
      for (int g = 0; g < 13; g += 2) {
        if (5 * g >= 3 * k) break;
        const uint32_t e = uint32_t(pid >> (5 * g)) & 31u;
        if (g < 12) screen_add2(x, table + g * kScreenGroupWords, e, uint32_t(pid >> (5 * g + 5)) & 31u);
        else screen_add(x, table + g * kScreenGroupWords, e);
      }
    } else {
      const uint32_t* group = table;
      uint64_t row = kRowStep;
      const auto coef = [&] {
        const uint32_t v = uint32_t(splitmix64(base ^ row)) & 7u;
        row += kRowStep;
        return v;
      };
      const auto add = [&](uint32_t m) {  // 15 bits
        screen_add2(x, group, m & 31u, (m >> 5) & 31u);
        screen_add(x, group + 2 * kScreenGroupWords, m >> 10);
        group += 3 * kScreenGroupWords;
      };
      int i = 0;
      for (; i + 5 <= k; i += 5) {
        uint32_t m = 0u;
#pragma unroll
        for (int j = 0; j < 5; ++j) m |= coef() << (3 * j);
        add(m);
      }
      if (i < k) {
        uint32_t m = 0u;
        for (int j = 0; i + j < k; ++j) m |= coef() << (3 * j);
        add(m);
      }
      // one coefficient is 1 where its hash gives 0
      const uint64_t xf = seed_forced ^ (wid * 0xA5A3564E27F8861Full);
      const uint32_t f = screen_mod(splitmix64(xf), uk, inv, r32);
      if ((uint32_t(splitmix64(base ^ (uint64_t(f + 1u) * kRowStep))) & 7u) == 0u) {
        const uint32_t g = 3u * f / 5u;
        screen_add(x, table + g * kScreenGroupWords, 1u << (3u * f - 5u * g));
      }
    }
    wmin = min(wmin, screen_weight(x));
    if (__any_sync(0xffffffffu, wmin < wthr || stop)) break;
  }
  wmin = __reduce_min_sync(0xffffffffu, wmin);
  if (lane == 0) {
    if (wmin < kN) atomicMax(a.out + c, kN - wmin);
    if (wmin < wthr) atomicExch(a.abort + c, 1);
  }
}

// Passes per CTA: up to 8, against the layout of a code's table (350 issue
// slots a warp; a pass has 250 at k = 16 and 900 at k = 30), as long as 32 CTAs
// per SM are left, for an even end; more only to keep the grid within bounds.
static cudaError_t launch_screen(const DistArgs& a, int sm_count, cudaStream_t s) {
  const uint64_t count = uint64_t(a.sample_count), n = uint64_t(a.n);
  const uint64_t rounds = count / kScreenThreads + (count % kScreenThreads != 0);
  const uint64_t fill = 32ull * uint64_t(sm_count);
  uint64_t passes = rounds >= 8ull * fill ? 8ull : std::min<uint64_t>(8ull, rounds * n / fill);
  passes = std::max<uint64_t>(passes, 1ull);
  const uint64_t most = std::max<uint64_t>((1ull << 30) / n, 1ull);  // pieces of a code
  passes = std::max(passes, (rounds + most - 1) / most);
  const uint64_t pieces = (rounds + passes - 1) / passes;
  screen_kernel<<<unsigned(pieces * n), kScreenThreads, screen_shared_bytes(a.k_max), s>>>(a,
                                                                                         passes);
  return cudaGetLastError();
}

}  // namespace tg
