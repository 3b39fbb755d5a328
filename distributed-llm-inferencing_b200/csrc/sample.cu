// Sampling epilogue: temperature -> top-k -> top-p -> multinomial, one cluster of CTAs per row.
//
// This is what the reference worker asks of generate() by default
// (worker/app.py:297-305: do_sample=True, top_k=50, top_p=0.95, temperature=0.8), i.e.
// TemperatureLogitsWarper -> TopKLogitsWarper -> TopPLogitsWarper -> softmax ->
// torch.multinomial (TF:generation/logits_process.py, TF:generation/utils.py:2762-2793),
// on the bf16 logits cast to fp32:
//   top-k keeps every logit >= the k-th largest (ties at the threshold are all kept, as
//         `scores < topk(scores, k)[0][..., -1]` does);
//   top-p keeps, in descending order of probability, the tokens whose EXCLUSIVE prefix sum
//         of (top-k-renormalised) probabilities is < top_p — the same set as HF's ascending
//         `cumsum <= 1 - top_p` removal — and always at least one token;
//   the draw is inverse-CDF over the kept tokens with a Philox4x32-10 uniform keyed by
//         (seed, step, row).  torch.multinomial uses a different stream and algorithm, so
//         draws agree in distribution, not bit for bit; the kept set and its probabilities
//         are what the parity test compares.
//
// What bounds it: latency.  A row is 64 ... 256 KB, a few us of one SM's load bandwidth, so it is cut over a cluster of up
// to 8 CTAs.  A CTA keeps the first 16 384 logits of its slice in registers, as keys that compare two at a time; what a longer
// slice has beyond them (many rows, fewer CTAs each) is read twice, for the bound and for the candidates.  The k-th largest logit
// is found without a histogram of the row: the k-th largest of a CTA's 512 per-thread maxima is a lower bound of it (k threads
// hold an element at least that large), the largest such bound of the cluster leaves a few hundred candidates, each CTA writes
// its own into its region of the first CTA's shared memory, and the exact threshold is a search over the bits in which bound and
// maximum differ.  Up to 64 that remain are put in order by counting and finished by one warp in registers; the uniform is drawn
// while the cluster meets.  One row of 128 256 logits takes 8.6 us, 48 rows 12.5.
// (The two 256-bin histograms with shared-memory atomics and their serial scans, three passes of 2-byte loads by one CTA per
// row, took 62 us for one row as for 48, V = 128 256.  They are left for large k, see launch_sample.)
#include <math.h>

#include "common.cuh"

namespace dli {

constexpr int kSampleThreads = 512;
constexpr int kMaxCand = 2048;  // candidates kept in shared memory (k plus ties)
constexpr int kMaxRanked = 128;  // candidates that are put in order by counting
constexpr int kOneWarp = 64;     // candidates that one warp finishes in registers

// monotone key: larger bf16 value <-> larger 16-bit key
__device__ __forceinline__ uint32_t bf16_key(uint16_t b) { return (b & 0x8000u) ? (uint16_t)~b : (uint16_t)(b | 0x8000u); }
__device__ __forceinline__ float key_value(uint32_t key) {
  const uint16_t b = (key & 0x8000u) ? (uint16_t)(key & 0x7fffu) : (uint16_t)~key;
  return __uint_as_float((uint32_t)b << 16);
}

struct Philox {
  uint32_t c[4], k[2];
  __device__ __forceinline__ static void mulhilo(uint32_t a, uint32_t b, uint32_t& hi, uint32_t& lo) {
    const uint64_t p = (uint64_t)a * b;
    hi = (uint32_t)(p >> 32);
    lo = (uint32_t)p;
  }
  __device__ __forceinline__ void round() {
    uint32_t h0, l0, h1, l1;
    mulhilo(0xD2511F53u, c[0], h0, l0);
    mulhilo(0xCD9E8D57u, c[2], h1, l1);
    const uint32_t n0 = h1 ^ c[1] ^ k[0], n1 = l1, n2 = h0 ^ c[3] ^ k[1], n3 = l0;
    c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
    k[0] += 0x9E3779B9u;
    k[1] += 0xBB67AE85u;
  }
};
// uniform in [0, 1) from Philox4x32-10 keyed by seed, counter (step, row)
__device__ __forceinline__ float philox_uniform(uint64_t seed, uint32_t step, uint32_t row) {
  Philox p;
  p.c[0] = step; p.c[1] = row; p.c[2] = 0x6a09e667u; p.c[3] = 0xbb67ae85u;
  p.k[0] = (uint32_t)seed; p.k[1] = (uint32_t)(seed >> 32);
#pragma unroll
  for (int i = 0; i < 10; ++i) p.round();
  return (float)(p.c[0] >> 8) * (1.0f / 16777216.0f);
}

// ---- clusters -----------------------------------------------------------------------------------------------------
constexpr int kSliceVecs = 4;                                  // 16-byte vectors a thread keeps in registers
constexpr int kSliceElems = kSampleThreads * kSliceVecs * 8;   // logits of a CTA that are read once
constexpr int kMaxRowCtas = 8;
constexpr int kRegionSlots = 8 * kSampleThreads;               // eight candidates a thread of the first CTA

__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p)), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_st(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_st16(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.b16 [%0], %1;" ::"r"(addr), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
  cluster_arrive();
  cluster_wait();
}

// bf16_key of both halves of a word.
__device__ __forceinline__ uint32_t bf16_keys2(uint32_t x) { return x ^ ((((x >> 15) & 0x00010001u) * 0x7fffu) | 0x80008000u); }
__device__ __forceinline__ uint4 bf16_keys8(const uint4& u) {
  return make_uint4(bf16_keys2(u.x), bf16_keys2(u.y), bf16_keys2(u.z), bf16_keys2(u.w));
}
__device__ __forceinline__ uint32_t max_keys2(uint32_t a, const uint4& u) {
  return __vmaxu2(__vmaxu2(a, __vmaxu2(u.x, u.y)), __vmaxu2(u.z, u.w));
}

// The largest t in [base, base + 2^bits) with at least k of the block's keys >= t, where k of them are >= base: a bit a step, a
// count of the block for each of a thread's first NQ keys (0.1 us; a test of how many there are inside the loop doubles that).
// Two bits a step take three counts, and every way to sum them over 16 warps (reductions, atomics) was slower: 0.28 us a step.
template <int NQ, int N>
__device__ __forceinline__ uint32_t kth_key(const uint32_t (&keys)[N], int k, uint32_t base, int bits) {
  uint32_t t = base;
#pragma unroll 1
  for (int sh = bits - 1; sh >= 0; --sh) {
    const uint32_t a = t + (1u << sh);
    int count = 0;
#pragma unroll
    for (int q = 0; q < NQ; ++q) count += __syncthreads_count(keys[q] >= a);
    if (count >= k) t = a;
  }
  return t;
}

// f(key, index) for every element of the row by the threads of one CTA, eight loads of a thread in flight at a time.
template <typename F>
__device__ __forceinline__ void for_each_key(const uint16_t* __restrict__ row, int V, F f) {
  constexpr int kBatch = 8;
  int i = threadIdx.x;
  for (; i + (kBatch - 1) * kSampleThreads < V; i += kBatch * kSampleThreads) {
    uint16_t raw[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) raw[u] = row[i + u * kSampleThreads];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) f(bf16_key(raw[u]), i + u * kSampleThreads);
  }
  for (; i < V; i += kSampleThreads) f(bf16_key(row[i]), i);
}

// Largest key t such that at least `k` elements of the row have key >= t (two 8-bit radix passes over global memory): the
// general form, for k above the number of threads and rows with more candidates than fit.
__device__ uint32_t kth_largest_key(const uint16_t* __restrict__ row, int V, int k, uint32_t* hist /*256*/,
                                    uint32_t* sh /*2*/) {
  const int tid = threadIdx.x;
  uint32_t prefix = 0;
  int remaining = k;
  for (int pass = 0; pass < 2; ++pass) {
    for (int i = tid; i < 256; i += kSampleThreads) hist[i] = 0;
    __syncthreads();
    for_each_key(row, V, [&](uint32_t key, int) {
      if (pass == 0) atomicAdd(&hist[key >> 8], 1u);
      else if ((key >> 8) == prefix) atomicAdd(&hist[key & 0xff], 1u);
    });
    __syncthreads();
    if (tid == 0) {
      int acc = 0, bin = 255;
      for (; bin > 0; --bin) {
        if (acc + (int)hist[bin] >= remaining) break;
        acc += hist[bin];
      }
      sh[0] = bin;
      sh[1] = remaining - acc;  // still needed inside this bin
    }
    __syncthreads();
    if (pass == 0) { prefix = sh[0]; remaining = sh[1]; }
    else prefix = (prefix << 8) | sh[0];
    __syncthreads();
  }
  return prefix;
}

// The candidates' order as whole numbers: larger value <-> larger number, -0 = 0, a NaN above every number; 0 lies below all.
__device__ __forceinline__ uint32_t order_key(float v) {
  const uint32_t u = __float_as_uint(v + 0.f);
  return v != v ? 0xffffffffu : (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float order_value(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
// Descending by value, equal values by ascending token id.
__device__ __forceinline__ bool comes_before(uint32_t a, int ia, uint32_t b, int ib) {
  return a > b || (a == b && (unsigned)ia < (unsigned)ib);
}

// grid: rows x CTAs of a row (a cluster).  narrow: see launch_sample; otherwise one CTA per row
__global__ void __launch_bounds__(kSampleThreads)
sample_kernel(const bf16* __restrict__ logits, int ld, int32_t* __restrict__ out, int V, float inv_temperature,
              int top_k, float top_p, const uint64_t* __restrict__ seed, const int32_t* __restrict__ step,
              float* __restrict__ dbg_probs, int32_t* __restrict__ dbg_ids, int dbg_cap, int per_row,
              const int32_t* __restrict__ row_mask, int ctas, int narrow) {
  __shared__ uint32_t hist[256];
  __shared__ uint32_t sh[2];
  __shared__ float cval[kMaxCand];  // candidates: keys, then values, then probabilities
  __shared__ int cidx[kMaxCand];
  __shared__ uint16_t gkey[kRegionSlots];  // first CTA: the row's candidates, a region per CTA of the cluster
  __shared__ int gidx[kRegionSlots];
  __shared__ uint32_t bounds[kMaxRowCtas];  // bound | largest key << 16 of each CTA
  __shared__ uint32_t counts[kMaxRowCtas];  // first CTA: candidates of each CTA
  __shared__ uint32_t tops[16], mths[16];   // of each warp: its largest key, its m-th largest maximum
  __shared__ int ncand;
  __shared__ int nties;
  __shared__ float uniform;
  __shared__ float red[kSampleThreads / 32];
  uint32_t* ckey = reinterpret_cast<uint32_t*>(cval);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b = blockIdx.x / ctas, rank = blockIdx.x - b * ctas;
  if (tid == 0) ncand = 0, nties = 0;
  pdl_wait();
  pdl_trigger();
  if (row_mask != nullptr && row_mask[b] == 0) return;  // this row keeps the token already in out[]
  const uint16_t* row = reinterpret_cast<const uint16_t*>(logits + (size_t)b * ld);
  const int k = top_k > 0 ? min(top_k, V) : V;
  // per_row: every row has its own (seed, step) and the row index stays out of the key, so a sequence's draws do not depend on
  // the batch row it happens to occupy.  One thread asks for the seed now and draws while the cluster meets.
  const bool drawer = rank == 0 && tid == 32;
  uint64_t my_seed = 0;
  uint32_t my_step = 0;
  if (drawer) {
    if (seed) my_seed = seed[per_row ? b : 0];
    if (step) my_step = (uint32_t)step[per_row ? b : 0];
  }

  int total = kMaxCand + 1;  // candidates of the row, if they fit
  const int per_region = kSampleThreads / ctas, region_slots = 8 * per_region;
  if (narrow) {
    // ---- this CTA's share of the row: whole 16-byte vectors; what lies before and after them goes to the first CTA --------
    const int head = min(V, (int)(((16u - (uint32_t)(reinterpret_cast<uintptr_t>(row) & 15u)) & 15u) >> 1));
    const int n_vec = (V - head) >> 3, tail0 = head + n_vec * 8;
    const int v0 = (int)((long long)n_vec * rank / ctas), v1 = (int)((long long)n_vec * (rank + 1) / ctas);
    const uint4* vecs = reinterpret_cast<const uint4*>(row + head);
    uint4 held[kSliceVecs];  // keys
#pragma unroll
    for (int i = 0; i < kSliceVecs; ++i) {
      const int v = v0 + i * kSampleThreads + tid;
      // beyond the slice: the lowest key (a negative NaN), never at or above a bound
      held[i] = v < v1 ? vecs[v] : make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
    }
    int edge = -1;  // an element of the unaligned ends
    if (rank == 0) {
      if (tid < head) edge = tid;
      else if (tail0 + tid - head < V) edge = tail0 + tid - head;
    }
    uint32_t top2 = 0;
#pragma unroll 4
    for (int v = v0 + kSliceVecs * kSampleThreads + tid; v < v1; v += kSampleThreads) top2 = max_keys2(top2, bf16_keys8(vecs[v]));
#pragma unroll
    for (int i = 0; i < kSliceVecs; ++i) {
      held[i] = bf16_keys8(held[i]);
      top2 = max_keys2(top2, held[i]);
    }
    uint32_t top[1] = {max(top2 & 0xffffu, top2 >> 16)};
    if (edge >= 0) top[0] = max(top[0], bf16_key(row[edge]));

    // ---- lower bound of the k-th largest key: the k-th largest of the per-thread maxima (a row of at most a thread per logit
    // needs none: all of it are candidates) ----
    uint32_t bound = 0, most = 0xffffu;
    cluster_arrive();
    if (V > kSampleThreads) {
      // It lies between the smallest and the largest of the 16 warps' m-th largest, m = k / 16 rounded up: at least 16 m of the
      // maxima reach the one, at most 16 (m - 1) < k exceed the other.  That leaves some 7 of the 16 bits.
      uint32_t v = top[0], mth = 0;
      for (int m = (k + 15) / 16, r = 1; r <= m; ++r) {
        mth = __reduce_max_sync(0xffffffffu, v);
        if (r == 1 && lane == 0) tops[warp] = mth;
        const unsigned holders = __ballot_sync(0xffffffffu, v == mth);
        if (lane == __ffs(holders) - 1) v = 0u;
      }
      if (lane == 0) mths[warp] = mth;
      __syncthreads();
      const uint32_t lo = __reduce_min_sync(0xffffffffu, mths[lane & 15]), hi = __reduce_max_sync(0xffffffffu, mths[lane & 15]);
      bound = kth_key<1>(top, k, lo, 32 - __clz(hi - lo));
      most = __reduce_max_sync(0xffffffffu, tops[lane & 15]);
    }
    cluster_wait();  // every CTA of the cluster runs: from here on its shared memory may be written
    if (tid < ctas) cluster_st(cluster_addr(&bounds[rank], tid), bound | most << 16);
    cluster_sync_all();
    most = 0;
    for (int c = 0; c < ctas; ++c) bound = max(bound, bounds[c] & 0xffffu), most = max(most, bounds[c] >> 16);
    // ---- candidates: this CTA's elements at or above the bound, straight into its region of the first CTA -------------------
    const uint32_t kb = cluster_addr(gkey, 0) + rank * region_slots * 2, ib = cluster_addr(gidx, 0) + rank * region_slots * 4;
    auto take = [&](uint32_t key, int i) {
      if (key >= bound) {
        const int slot = atomicAdd(&ncand, 1);
        if (slot < region_slots) {
          cluster_st16(kb + slot * 2, key);
          cluster_st(ib + slot * 4, (uint32_t)i);
        }
      }
    };
    const uint32_t bound2 = bound | bound << 16;
    auto take8 = [&](const uint4& u, int i) {
      const uint32_t top8 = max_keys2(0u, u);
      if (max(top8 & 0xffffu, top8 >> 16) < bound) return;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t w = e == 0 ? u.x : e == 1 ? u.y : e == 2 ? u.z : u.w;
        if (__vmaxu2(w, bound2) == bound2 && (w & 0xffffu) != bound && (w >> 16) != bound) continue;
        take(w & 0xffffu, i + 2 * e);
        take(w >> 16, i + 2 * e + 1);
      }
    };
#pragma unroll
    for (int i = 0; i < kSliceVecs; ++i) {
      const int v = v0 + i * kSampleThreads + tid;
      if (v < v1) take8(held[i], head + v * 8);
    }
#pragma unroll 4
    for (int v = v0 + kSliceVecs * kSampleThreads + tid; v < v1; v += kSampleThreads) take8(bf16_keys8(vecs[v]), head + v * 8);
    if (edge >= 0) take(bf16_key(row[edge]), edge);
    __syncthreads();
    if (tid == 0) cluster_st(cluster_addr(&counts[rank], 0), (uint32_t)ncand);
    cluster_arrive();
    if (drawer) uniform = philox_uniform(my_seed, my_step, per_row ? 0u : b);
    __syncwarp();
    cluster_wait();
    if (rank != 0) return;

    // ---- first CTA: the exact threshold, and everything at or above it (ties are kept) --------------------------------
    uint32_t fullest = 0;
    total = 0;
    for (int c = 0; c < ctas; ++c) total += counts[c], fullest = max(fullest, counts[c]);
    if (tid == 0) ncand = 0;
    if (fullest <= (uint32_t)region_slots && total <= kMaxCand) {
      const int region = tid / per_region, at = tid - region * per_region;
      const int mine = region < ctas ? (int)counts[region] : 0;
      const int nq = ((int)fullest + per_region - 1) / per_region;  // at most 8
      uint32_t keys[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        keys[q] = q < nq && q * per_region + at < mine ? gkey[region * region_slots + q * per_region + at] : 0u;
      const int bits = 32 - __clz(most - bound);
      const uint32_t thr = nq == 1   ? kth_key<1>(keys, k, bound, bits)
                           : nq == 2 ? kth_key<2>(keys, k, bound, bits)
                           : nq == 3 ? kth_key<3>(keys, k, bound, bits)
                           : nq == 4 ? kth_key<4>(keys, k, bound, bits)
                                     : kth_key<8>(keys, k, bound, bits);  // keys past the counted ones are 0
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (q >= nq) break;
        const bool in = q * per_region + at < mine && keys[q] >= thr;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        int first = 0;
        if (m && lane == 0) first = atomicAdd(&ncand, __popc(m));
        first = __shfl_sync(0xffffffffu, first, 0);
        if (in) {
          const int slot = first + __popc(m & ((1u << lane) - 1));
          ckey[slot] = order_key(key_value(keys[q]) * inv_temperature);
          cidx[slot] = gidx[region * region_slots + q * per_region + at];
        }
      }
    } else {
      total = kMaxCand + 1;
    }
  } else if (drawer) {
    uniform = philox_uniform(my_seed, my_step, per_row ? 0u : b);
  }
  if (total > kMaxCand) {
    __syncthreads();
    const uint32_t thr = kth_largest_key(row, V, min(k, kMaxCand), hist, sh);
    // what lies above the threshold (fewer than k elements) first: ties beyond the capacity are dropped, never those
    for_each_key(row, V, [&](uint32_t key, int i) {
      if (key > thr) {
        const int slot = atomicAdd(&ncand, 1);
        ckey[slot] = order_key(key_value(key) * inv_temperature);
        cidx[slot] = i;
      } else if (key == thr) {
        const int slot = atomicAdd(&nties, 1);
        if (slot < kMaxCand) gidx[slot] = i;
      }
    });
    __syncthreads();
    const int above = ncand, ties = min(nties, kMaxCand - above);
    __syncthreads();
    for (int i = tid; i < ties; i += kSampleThreads) {
      ckey[above + i] = order_key(key_value(thr) * inv_temperature);
      cidx[above + i] = gidx[i];
    }
    if (tid == 0) ncand = above + ties;
  }
  __syncthreads();
  const int n = ncand;  // at most kMaxCand
  if (n <= kOneWarp) {
    // A few: each one's place is the number of those before it, counted by eight threads; one warp does the rest in registers.
    // The sums are formed in the order of the general form below.
    const int me = tid >> 3;
    const uint32_t a = ckey[min(me, n - 1)];
    const int ia = cidx[min(me, n - 1)];
    int place = 0;
    for (int j = tid & 7; j < n; j += 8) place += comes_before(ckey[j], cidx[j], a, ia) ? 1 : 0;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) place += __shfl_xor_sync(0xffffffffu, place, o);
    uint32_t* const skey = ckey + kOneWarp;
    int* const sidx = cidx + kOneWarp;
    if (me < n && (tid & 7) == 0) skey[place] = a, sidx[place] = ia;
    __syncthreads();
    if (warp != 0) return;
    const float vmax = order_value(skey[0]);
    float p[2], sum[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      p[h] = h * 32 + lane < n ? __expf(order_value(skey[h * 32 + lane]) - vmax) : 0.f;
      sum[h] = warp_sum(p[h]);
    }
    const float denom = sum[0] + sum[1];
    int kept = 0;
    float carry = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      p[h] /= denom;
      float incl = p[h];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      const int i = h * 32 + lane;
      const unsigned m = __ballot_sync(0xffffffffu, i < n && (i == 0 || carry + incl - p[h] < top_p));
      if (kept == h * 32) kept += __popc(m);
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    kept = max(kept, 1);
    float mass = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (h * 32 + lane < kept) mass += p[h];
    mass = warp_sum(mass);
    if (dbg_probs) {
      for (int i = lane; i < dbg_cap; i += 32) {
        dbg_probs[(size_t)b * dbg_cap + i] = i < kept ? (i < 32 ? p[0] : p[1]) / mass : 0.f;
        dbg_ids[(size_t)b * dbg_cap + i] = i < kept ? sidx[i] : -1;
      }
    }
    // the inverse CDF, its sums in order: every lane walks them
    const float u = uniform * mass;
    float acc = 0.f;
    int pick = kept - 1;
#pragma unroll
    for (int i0 = 0; i0 < 64; i0 += 8) {
      if (i0 >= kept) break;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        acc += __shfl_sync(0xffffffffu, p[i0 >> 5], (i0 & 31) + e);
        if (i0 + e < pick && u < acc) pick = i0 + e;
      }
      if (u < acc) break;
    }
    if (lane == 0) out[b] = sidx[pick];
    return;
  }
  // Descending by value, equal values by ascending token id.  Which of several EQUAL-probability tokens survive at the
  // nucleus boundary depends on torch.sort's tie order in the reference (not specified); here the lower token ids stay.
  int npow = 1;
  while (npow < n) npow <<= 1;
  if (n == 1) {
    // in order already
  } else if (npow <= kMaxRanked) {
    // every candidate's place is the number of those before it, counted by `lanes` threads of a warp (500 candidates counted
    // by one thread each took 30 us, the sorting network takes 4)
    const int lanes = min(32, kSampleThreads / npow), me = tid / lanes;
    const uint32_t a = ckey[min(me, n - 1)];
    const int ia = cidx[min(me, n - 1)];
    int place = 0;
    for (int j = tid % lanes; j < n; j += lanes) place += comes_before(ckey[j], cidx[j], a, ia) ? 1 : 0;
    for (int o = lanes >> 1; o > 0; o >>= 1) place += __shfl_xor_sync(0xffffffffu, place, o);
    __syncthreads();
    if (me < n && tid % lanes == 0) { ckey[place] = a; cidx[place] = ia; }
    __syncthreads();
  } else {
    for (int i = n + tid; i < npow; i += kSampleThreads) { ckey[i] = 0u; cidx[i] = -1; }
    __syncthreads();
    // bitonic sort
    for (int size = 2; size <= npow; size <<= 1) {
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int i = tid; i < npow; i += kSampleThreads) {
          const int j = i ^ stride;
          if (j > i) {
            const bool desc = (i & size) == 0;
            const uint32_t a = ckey[i], b = ckey[j];
            const int ia = cidx[i], ib = cidx[j];
            if (comes_before(a, ia, b, ib) != desc) { ckey[i] = b; ckey[j] = a; cidx[i] = ib; cidx[j] = ia; }
          }
        }
        __syncthreads();
      }
    }
  }
  // ---- softmax over the top-k set, nucleus cut, renormalise, draw (n <= 2048: one warp scans) ----
  const float vmax = order_value(ckey[0]);
  float part = 0.f;
  for (int i = tid; i < n; i += kSampleThreads) part += __expf(order_value(ckey[i]) - vmax);
  part = warp_sum(part);
  if (lane == 0) red[warp] = part;
  __syncthreads();
  float denom = 0.f;
#pragma unroll
  for (int w = 0; w < kSampleThreads / 32; ++w) denom += red[w];
  for (int i = tid; i < n; i += kSampleThreads) cval[i] = __expf(order_value(ckey[i]) - vmax) / denom;  // probabilities, descending
  __syncthreads();
  if (warp == 0) {
    // exclusive prefix sums in descending order; keep while prefix < top_p (always the first)
    float carry = 0.f;
    int kept = 0;
    for (int base = 0; base < n; base += 32) {
      const int i = base + lane;
      const float p = i < n ? cval[i] : 0.f;
      float incl = p;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      const float excl = carry + incl - p;
      const bool keep = i < n && (i == 0 || excl < top_p);
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      kept += __popc(m);
      carry += __shfl_sync(0xffffffffu, incl, 31);
      if (m != 0xffffffffu) break;
    }
    kept = max(kept, 1);
    float mass = 0.f;
    for (int i = lane; i < kept; i += 32) mass += cval[i];
    mass = warp_sum(mass);
    if (dbg_probs) {
      for (int i = lane; i < dbg_cap; i += 32) {
        dbg_probs[(size_t)b * dbg_cap + i] = i < kept ? cval[i] / mass : 0.f;
        dbg_ids[(size_t)b * dbg_cap + i] = i < kept ? cidx[i] : -1;
      }
    }
    if (lane == 0) {
      const float u = uniform * mass;
      float acc = 0.f;
      int pick = kept - 1;
      for (int i0 = 0; i0 < kept; i0 += 8) {  // eight loads in flight, the sums in order
        float p[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) p[e] = cval[min(i0 + e, kept - 1)];
        int first = kept;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          acc += p[e];
          if (first == kept && i0 + e < kept && u < acc) first = i0 + e;
        }
        if (first < kept) { pick = first; break; }
      }
      out[b] = cidx[pick];
    }
  }
}

// CTAs that run at once as clusters of 1 ... 8 (asked of the driver once per device).
static int sample_capacity(int* capacity /*[kMaxRowCtas + 1]*/) {
  static PerDeviceOnce once;
  static int cap[kMaxDevices][kMaxRowCtas + 1];
  DLI_ONCE_PER_DEVICE(once, dev, {
    for (int c = 1; c <= kMaxRowCtas; ++c) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)c * 1024);
      cfg.blockDim = dim3(kSampleThreads);
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = c;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int n = 0;
      DLI_CUDA_CALL(cudaOccupancyMaxActiveClusters(&n, sample_kernel, &cfg));
      cap[dev][c] = n * c;
    }
  });
  for (int c = 1; c <= kMaxRowCtas; ++c) capacity[c] = cap[dev][c];
  return DLI_OK;
}

// A cluster of as many CTAs as the row has slices of 16 384 logits, at most the portable 8, and no more than let all rows'
// clusters run at once (two CTAs share an SM: clusters of 8 / 5 / 4 / 2 hold 264 / 270 / 280 / 296 CTAs at once): a second wave is a
// second chain, a longer slice a few loads.  128 256 logits, us with 8 / 5 / 4 / 2 / 1 CTAs a row: one row 8.5 / 10.0 / 10.7 / 12.8 /
// 17.5, 24 rows 10.7 / 11.0 / 11.9 / 13.9 / 18.0, 48 rows 16.8 / 12.4 / 13.8 / 14.3 / 18.2, 64 rows 20.1 / 19.3 / 13.7 / 15.0 / 18.5,
// 128 rows 33.5 / 27.1 / 25.8 / 17.4 / 19.7: what the rule takes is the fastest of all eight sizes in each line.
// That way (`narrow`) is for k small enough that few logits lie above the bound: with `per` logits a thread, k of 512 maxima above
// it means a share of 1 - (1 - k/512)^(1/per) of all logits, and a bf16 step at the bound adds up to some V / 4096 ties.  Larger
// k would overflow the first CTA's shared memory after all the work; it takes the histograms of one CTA per row at once.
//   one row, us, one CTA for every k / clusters up to k = 512 / this rule: 128 256 logits, k = 128: 62.3 / 21.0 / 17.3,
//   k = 256: 65.5 / 109 / 65.1, k = 512: 76.2 / 107 / 74.5, k = 1000: 97.3 / 105 / 79.2; 500 logits, k = 500: 16.3 / 47.9 / 15.7
static int launch_sample(const char* what, const void* logits, int ld, int32_t* out, int B, int V, float temperature,
                         int top_k, float top_p, const uint64_t* seed, const int32_t* step, float* dbg_probs,
                         int32_t* dbg_ids, int dbg_cap, int per_row, const int32_t* row_mask, cudaStream_t s) {
  int ctas = (V - 1) / kSliceElems + 1;
  if (ctas > kMaxRowCtas) ctas = kMaxRowCtas;
  int cap[kMaxRowCtas + 1];
  const int rc = sample_capacity(cap);
  if (rc != DLI_OK) return rc;
  while (ctas > 1 && (long long)B * ctas > cap[ctas]) --ctas;
  const int k = top_k > 0 && top_k < V ? top_k : V;
  const double per = (double)V / (kSampleThreads * ctas);
  const bool narrow = k <= kSampleThreads &&
                      (V <= kMaxCand || V * (1.0 - pow(1.0 - (double)k / kSampleThreads, 1.0 / per)) <= kMaxCand - V / 4096);
  if (!narrow) ctas = 1;
  const cudaError_t e = launch_kernel_cluster(sample_kernel, dim3((unsigned)B * ctas), dim3(kSampleThreads), (size_t)0, s,
                                              (unsigned)ctas, (const bf16*)logits, ld, out, V, 1.0f / temperature, top_k,
                                              top_p, seed, step, dbg_probs, dbg_ids, dbg_cap, per_row, row_mask, ctas,
                                              narrow ? 1 : 0);
  if (e != cudaSuccess) return fail(DLI_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  return DLI_OK;
}

}  // namespace dli

extern "C" int dli_sample_bf16(const void* logits, int ld, int32_t* out, int B, int V, float temperature, int top_k,
                               float top_p, const uint64_t* seed, const int32_t* step, float* dbg_probs,
                               int32_t* dbg_ids, int dbg_cap, dli_stream_t stream) {
  using namespace dli;
  DLI_CHECK_ARG(logits && out, "dli_sample_bf16: null pointer");
  DLI_CHECK_ARG(B >= 0 && V > 0 && ld >= V, "dli_sample_bf16: bad sizes B=%d V=%d ld=%d", B, V, ld);
  DLI_CHECK_ARG(temperature > 0.f && top_p > 0.f && top_p <= 1.f && top_k >= 0,
                "dli_sample_bf16: need temperature > 0, 0 < top_p <= 1, top_k >= 0 (0 = off)");
  DLI_CHECK_ARG((top_k > 0 && top_k <= kMaxCand) || V <= kMaxCand,
                "dli_sample_bf16: top_k must be 1..%d when the vocabulary is larger than that", kMaxCand);
  DLI_CHECK_ARG((dbg_probs == nullptr) == (dbg_ids == nullptr) && dbg_cap >= 0, "dli_sample_bf16: bad debug buffers");
  if (B == 0) return DLI_OK;
  return launch_sample("dli_sample_bf16", logits, ld, out, B, V, temperature, top_k, top_p, seed, step, dbg_probs, dbg_ids,
                       dbg_cap, 0, nullptr, static_cast<cudaStream_t>(stream));
}

extern "C" int dli_sample_rows_bf16(const void* logits, int ld, int32_t* out, int B, int V, float temperature,
                                    int top_k, float top_p, const uint64_t* seeds, const int32_t* steps,
                                    const int32_t* row_mask, dli_stream_t stream) {
  using namespace dli;
  DLI_CHECK_ARG(logits && out && seeds && steps, "dli_sample_rows_bf16: null pointer");
  DLI_CHECK_ARG(B >= 0 && V > 0 && ld >= V, "dli_sample_rows_bf16: bad sizes B=%d V=%d ld=%d", B, V, ld);
  DLI_CHECK_ARG(temperature > 0.f && top_p > 0.f && top_p <= 1.f && top_k >= 0,
                "dli_sample_rows_bf16: need temperature > 0, 0 < top_p <= 1, top_k >= 0 (0 = off)");
  DLI_CHECK_ARG((top_k > 0 && top_k <= kMaxCand) || V <= kMaxCand,
                "dli_sample_rows_bf16: top_k must be 1..%d when the vocabulary is larger than that", kMaxCand);
  if (B == 0) return DLI_OK;
  return launch_sample("dli_sample_rows_bf16", logits, ld, out, B, V, temperature, top_k, top_p, seeds, steps, nullptr,
                       nullptr, 0, 1, row_mask, static_cast<cudaStream_t>(stream));
}
