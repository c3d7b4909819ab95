// AGL2(F7) canonical forms of exponent sets and a device hash set for
// canonical dedup.
//
// Canonical form (the reference's canonical_forms kernel, kernel_canon.py:44-129,
// and canonical_forms_batch, champion_search_canonical.py:115-140): the
// minimum over A in GL2(F7) and anchor s in S of sort(A.S - A.s), packed 6 bits
// per index with the largest index most significant.  For sets of equal size
// that order is the order of 49-bit masks (bit i = exponent index i), so the
// key is the smallest mask among the AGL2 images of S that contain the origin.
// This file computes that mask for any popcount 1..49 (canon_form.cuh) and
// derives the reference's packed 128-bit key from it for k <= 16.
#include "common.cuh"
#include "canon_form.cuh"
#include "canonical.cuh"

namespace tg {

// 16 sets per CTA (8 lanes each): 64 sets already spread over 4 SMs, and the
// tables and lists take 8 KB of shared memory, so registers bound the
// occupancy.
constexpr int kCanonTPB = 128;
constexpr int kCanonSets = kCanonTPB / 8;

struct CanonArgs {
  const int32_t* sets;    // (n, k) rows, or NULL
  const uint64_t* masks;  // n masks when sets == NULL (parents when expand)
  int expand;             // set s = parent s / 49 plus point s % 49 (0 if present)
  int n;
  int k;
  uint64_t* out_mask;
  uint64_t* out_lo;
  uint64_t* out_hi;
  int32_t* status;
};

__global__ void __launch_bounds__(kCanonTPB) canon_kernel(CanonArgs a) {
  __shared__ CanonTable tab;
  __shared__ CanonScratch scratch[kCanonTPB / 32];
  {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(&g_canon_table);
    uint32_t* dst = reinterpret_cast<uint32_t*>(&tab);
    for (int i = threadIdx.x; i < int(sizeof(CanonTable) / 4); i += kCanonTPB) dst[i] = src[i];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int d = lane & 7;
  // The warp's first set decides, so all 32 lanes stay in the loop.
  for (int first = blockIdx.x * kCanonSets + (threadIdx.x >> 5) * 4; first < a.n;
       first += gridDim.x * kCanonSets) {
    const int s = first + (lane >> 3);
    uint64_t S = 0ull;
    bool bad = false;
    if (s < a.n) {
      if (a.sets) {
        const int32_t* row = a.sets + size_t(s) * size_t(a.k);
        for (int i = d; i < a.k; i += 8) {
          const int x = row[i];
          if (x < 0 || x >= kN) bad = true;
          else S |= 1ull << x;
        }
      } else if (a.expand) {
        const uint64_t parent = a.masks[s / kN] & kMask49;
        const int p = s % kN;
        S = (parent >> p & 1ull) ? 0ull : (parent | (1ull << p));
      } else {
        S = a.masks[s] & kMask49;
      }
    }
    if (a.sets) {
      // the lanes' points joined; a repeated index leaves fewer than k
      for (int o = 4; o > 0; o >>= 1) {
        S |= __shfl_xor_sync(0xffffffffu, S, o);
        bad |= __shfl_xor_sync(0xffffffffu, int(bad), o) != 0;
      }
      bad |= s < a.n && __popcll(S) != a.k;
    }
    if (bad) S = 0ull;
    const uint64_t best = canon_mask_groups(lane, S, tab, scratch[threadIdx.x >> 5]);
    if (d == 0 && s < a.n) {
      if (S == 0ull) {
        a.out_mask[s] = 0ull;
        if (a.out_lo) a.out_lo[s] = ~0ull;
        if (a.out_hi) a.out_hi[s] = ~0ull;
        if (bad && a.status) atomicCAS(a.status, 0, TG_ERR_BAD_INPUT);
      } else {
        a.out_mask[s] = best;
        if (a.out_lo || a.out_hi) {
          uint64_t lo, hi;
          key_from_mask(best, lo, hi);
          if (a.out_lo) a.out_lo[s] = lo;
          if (a.out_hi) a.out_hi[s] = hi;
        }
      }
    }
  }
}

int run_canonical(int sm_count, const int32_t* d_sets, const uint64_t* d_masks, int n, int k,
                  uint64_t* d_out_mask, uint64_t* d_lo, uint64_t* d_hi, int32_t* d_status,
                  cudaStream_t s, int expand) {
  if (n <= 0) return TG_OK;
  CanonArgs a{d_sets, d_masks, expand, n, k, d_out_mask, d_lo, d_hi, d_status};
  const int grid = min((n + kCanonSets - 1) / kCanonSets, sm_count * 16);
  canon_kernel<<<grid, kCanonTPB, 0, s>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "canon_kernel launch");
  return TG_OK;
}

// ---------------------------------------------------------------------------
// Device hash set: open addressing, linear probing, 64-bit keys.
// Layout: [256-byte header][keys: cap x u64][tags: cap x u64].
// A tag is (call_id << 32 | index of first insertion in that call); the
// smallest tag wins, so old keys stay old and within a call the first index
// is the representative, whatever the thread order.
// ---------------------------------------------------------------------------

constexpr uint64_t kEmpty = ~0ull;

struct HashHeader {
  unsigned long long count;  // occupied slots
};

__device__ __forceinline__ uint64_t hash_slot(uint64_t key, uint64_t cap) {
  return splitmix64(key) & (cap - 1ull);
}

__global__ void hash_clear_kernel(uint64_t* keys, uint64_t* tags, uint64_t cap, HashHeader* h) {
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < cap; i += stride) {
    keys[i] = kEmpty;
    tags[i] = kEmpty;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) h->count = 0ull;
}

__global__ void hash_insert_kernel(uint64_t* keys, uint64_t* tags, uint64_t cap, HashHeader* h,
                                   const uint64_t* in, int n, uint32_t call_id, int32_t* status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t key = in[i];
  if (key == kEmpty || key == 0ull) return;  // not a key: never new
  const unsigned long long tag = (static_cast<unsigned long long>(call_id) << 32) | uint32_t(i);
  uint64_t slot = hash_slot(key, cap);
  for (uint64_t probe = 0; probe < cap; ++probe) {
    const unsigned long long old = atomicCAS(reinterpret_cast<unsigned long long*>(keys + slot),
                                             static_cast<unsigned long long>(kEmpty),
                                             static_cast<unsigned long long>(key));
    if (old == kEmpty || old == key) {
      if (old == kEmpty) {
        const unsigned long long cnt = atomicAdd(&h->count, 1ull) + 1ull;
        if (cnt > cap / 2 && status) atomicCAS(status, 0, TG_ERR_CAPACITY);
      }
      atomicMin(reinterpret_cast<unsigned long long*>(tags + slot), tag);
      return;
    }
    slot = (slot + 1ull) & (cap - 1ull);
  }
  if (status) atomicCAS(status, 0, TG_ERR_CAPACITY);
}

__global__ void hash_mark_kernel(const uint64_t* keys, const uint64_t* tags, uint64_t cap,
                                 const uint64_t* in, int n, uint32_t call_id, uint8_t* is_new,
                                 int32_t* n_new) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool fresh = false;
  if (i < n) {
    const uint64_t key = in[i];
    if (key != kEmpty && key != 0ull) {
      const unsigned long long tag = (static_cast<unsigned long long>(call_id) << 32) | uint32_t(i);
      uint64_t slot = hash_slot(key, cap);
      for (uint64_t probe = 0; probe < cap; ++probe) {
        const uint64_t k = keys[slot];
        if (k == key) {
          fresh = tags[slot] == tag;
          break;
        }
        if (k == kEmpty) break;
        slot = (slot + 1ull) & (cap - 1ull);
      }
    }
    if (is_new) is_new[i] = fresh ? 1 : 0;
  }
  if (n_new) {
    const unsigned b = __ballot_sync(0xffffffffu, fresh);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(n_new, __popc(b));
  }
}

size_t hashset_bytes(int64_t cap) { return 256 + size_t(cap) * 16; }

// ---------------------------------------------------------------------------
// Order-preserving compaction of flagged masks into sorted index rows.
// ---------------------------------------------------------------------------

constexpr int kCompactTPB = 256;

__global__ void compact_count_kernel(const uint8_t* flags, int n, int* block_counts) {
  __shared__ int s_cnt;
  if (threadIdx.x == 0) s_cnt = 0;
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool f = i < n && flags[i];
  const unsigned b = __ballot_sync(0xffffffffu, f);
  if ((threadIdx.x & 31) == 0 && b) atomicAdd(&s_cnt, __popc(b));
  __syncthreads();
  if (threadIdx.x == 0) block_counts[blockIdx.x] = s_cnt;
}

__global__ void compact_scan_kernel(int* block_counts, int nb, int* total) {
  // one thread: the number of blocks is n / 256 (a few tens of thousands)
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    int run = 0;
    for (int b = 0; b < nb; ++b) {
      const int c = block_counts[b];
      block_counts[b] = run;
      run += c;
    }
    *total = run;
  }
}

__global__ void compact_write_kernel(const uint64_t* masks, const uint8_t* flags, int n, int k,
                                     const int* block_offsets, uint64_t* out_masks,
                                     int32_t* out_sets, int64_t* out_offsets) {
  __shared__ int s_warp[kCompactTPB / 32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool f = i < n && flags[i];
  const unsigned b = __ballot_sync(0xffffffffu, f);
  if (lane == 0) s_warp[w] = __popc(b);
  __syncthreads();
  int before = block_offsets[blockIdx.x];
  for (int j = 0; j < w; ++j) before += s_warp[j];
  before += __popc(b & ((1u << lane) - 1u));
  if (f) {
    const uint64_t m = masks[i];
    if (out_masks) out_masks[before] = m;
    if (out_sets) {
      int32_t* row = out_sets + size_t(before) * size_t(k);
      uint64_t x = m;
      for (int j = 0; j < k; ++j) {
        const int idx = x ? __ffsll(static_cast<long long>(x)) - 1 : 0;
        x &= x - 1ull;
        row[j] = idx;
      }
    }
    if (out_offsets) {
      out_offsets[before] = int64_t(before) * k;
      out_offsets[before + 1] = int64_t(before + 1) * k;
    }
  }
}

size_t compact_scratch_bytes(int n) {
  return size_t((n + kCompactTPB - 1) / kCompactTPB + 1) * sizeof(int);
}

int run_compact(const uint64_t* d_masks, const uint8_t* d_flags, int n, int k, void* d_scratch,
                uint64_t* d_out_masks, int32_t* d_out_sets, int64_t* d_out_offsets,
                int32_t* d_count, cudaStream_t s) {
  if (n <= 0) {
    cudaError_t e = cudaMemsetAsync(d_count, 0, sizeof(int32_t), s);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(count)");
    if (d_out_offsets) {
      e = cudaMemsetAsync(d_out_offsets, 0, sizeof(int64_t), s);
      if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(offsets)");
    }
    return TG_OK;
  }
  const int nb = (n + kCompactTPB - 1) / kCompactTPB;
  int* counts = static_cast<int*>(d_scratch);
  compact_count_kernel<<<nb, kCompactTPB, 0, s>>>(d_flags, n, counts);
  compact_scan_kernel<<<1, 32, 0, s>>>(counts, nb, d_count);
  if (d_out_offsets) {
    cudaError_t e = cudaMemsetAsync(d_out_offsets, 0, sizeof(int64_t), s);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(offsets)");
  }
  compact_write_kernel<<<nb, kCompactTPB, 0, s>>>(d_masks, d_flags, n, k, counts, d_out_masks,
                                                   d_out_sets, d_out_offsets);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "compact kernels launch");
  return TG_OK;
}

int run_hash_clear(void* table, int64_t cap, cudaStream_t s) {
  uint8_t* base = static_cast<uint8_t*>(table);
  uint64_t* keys = reinterpret_cast<uint64_t*>(base + 256);
  uint64_t* tags = keys + cap;
  HashHeader* h = reinterpret_cast<HashHeader*>(base);
  int grid = int((cap + 255) / 256);
  if (grid > 4096) grid = 4096;
  hash_clear_kernel<<<grid, 256, 0, s>>>(keys, tags, uint64_t(cap), h);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "hash_clear_kernel launch");
  return TG_OK;
}

int run_hash_insert(void* table, int64_t cap, const uint64_t* d_keys, int n, uint32_t call_id,
                    uint8_t* d_is_new, int32_t* d_n_new, int32_t* d_status, cudaStream_t s) {
  if (n <= 0) {
    if (d_n_new) {
      cudaError_t e = cudaMemsetAsync(d_n_new, 0, sizeof(int32_t), s);
      if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(n_new)");
    }
    return TG_OK;
  }
  uint8_t* base = static_cast<uint8_t*>(table);
  uint64_t* keys = reinterpret_cast<uint64_t*>(base + 256);
  uint64_t* tags = keys + cap;
  HashHeader* h = reinterpret_cast<HashHeader*>(base);
  if (d_n_new) {
    cudaError_t e = cudaMemsetAsync(d_n_new, 0, sizeof(int32_t), s);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(n_new)");
  }
  const int grid = (n + 255) / 256;
  hash_insert_kernel<<<grid, 256, 0, s>>>(keys, tags, uint64_t(cap), h, d_keys, n, call_id, d_status);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "hash_insert_kernel launch");
  hash_mark_kernel<<<grid, 256, 0, s>>>(keys, tags, uint64_t(cap), d_keys, n, call_id, d_is_new,
                                        d_n_new);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "hash_mark_kernel launch");
  return TG_OK;
}

}  // namespace tg
