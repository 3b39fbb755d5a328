// bf16 projections of many rows on pairs of SMs: tcgen05.mma.cta_group::2.
//
//   y[M,N] = epi( x[M,K] . w[N,K]^T )
//
// The two CTAs of a cluster share a tile of 256 activation rows x `bn` weight rows: each loads its own 128 activation rows and
// HALF of the weight rows, the leader's MMA reads both shared memories, and each CTA's TMEM holds the sums of its own rows (two
// stages of up to 256 columns, so the epilogue runs under the next tile's MMAs).  Per MMA an SM's shared memory takes in and
// gives out 8 KB instead of the 12 KB of a 128 x 256 tile on one SM, and the tile asks L2 for a third less.  Persistent, one
// CTA per SM: warp 0 = TMA producer, warp 1 of the leader = MMA issuer, warps 2-9 = epilogue.
//
// What bounds it: at 4 096 rows the tensor pipe, busy 93 % of the time under the power limit (28672 x 4096 gated: 588 us by itself,
// 709 us at 1.29 GHz after a second of nothing else, 1 357 TFLOP/s; profiles/pairs_notes.md); below some 1 000 rows whole rounds
// of tiles, which the width and a tail of narrower tiles even out (pair_cost); at K = 768 ... 2048 what no tile hides: 2.5 us from
// the predecessor's end to the first load, the last epilogue.
// Measured on B200 in chains of launches over rotating weights, in turn with the other kernels, us, 128-row tiles on single SMs /
// clusters (gemm_rows.cu) / here:
//   rows            301              450              1024             1777             4096
//   6144 x 4096      39 /  25 /  24   40 /  29 /  25   55 /  55 /  36   85 /  79 /  60  173 / 219 / 134
//   4096 x 4096      32 /  19 /  18   32 /  21 /  18   33 /  33 /  25   53 /  60 /  40  117 / 149 /  92
//   4096 x 14336     91 /  40 /  50   90 /  60 /  51   98 / 106 /  81  161 / 184 / 143  380 / 464 / 360
//   28672 gated      84 /  76 /  82  113 / 119 /  91  188 / 247 / 165  323 / 410 / 291  711 / 926 / 647
//   2048 x 5632      39 /  15 /  20   39 /  18 /  20   39 /  25 /  21   40 /  36 /  29   73 /  86 /  64
//   768 x 3072       26 /   8 /  11   26 /   9 /  11   25 /  12 /  12   26 /  15 /  13   25 /  22 /  16
#include "cta_pair.cuh"
#include "gemm_pair.cuh"
#include "recent.h"

namespace dli {

constexpr int kPairThreads = 64 + 8 * 32;  // TMA warp, MMA warp, eight epilogue warps (two per TMEM lane quadrant)
constexpr int kPairMaxStages = 8;
constexpr int kPairABytes = 128 * kBlockK * 2;
constexpr int kPairAccCols = 256;  // TMEM columns per accumulator stage, two stages
constexpr int kPairStageBytes = 32 * 128;  // an epilogue warp's line buffer: 32 rows x 64 bf16
constexpr int kPairSmemMax = 227 * 1024;
constexpr int kPairSmemFixed = 1024 + 8 * kPairStageBytes + 256;  // alignment, line buffers, barriers

__device__ __forceinline__ uint32_t pair_bias(const bf16* b) {  // two of them, from any address
  return (uint32_t)__bfloat16_as_ushort(b[0]) | ((uint32_t)__bfloat16_as_ushort(b[1]) << 16);
}

// What tile number `t` is: rows from m0, weight rows from n0 (in rows of w), `width` of them.  The first n_main * bn weight
// rows go in tiles of bn, the rest in tiles of bn_tail.  Row tiles in groups of 8, in a group rows fastest: the pairs in
// flight cover about 8 x 9 tiles, so both operands are used again out of L2.
struct PairTile { int m0, n0, width; };
__device__ __forceinline__ PairTile pair_tile(int t, int m_tiles, int n_main, int bn, int bn_tail, int n_tiles) {
  constexpr int kGroup = 8;
  const int main = m_tiles * n_main;
  const bool tail = t >= main;
  if (tail) t -= main;
  const int cols = tail ? n_tiles - n_main : n_main;
  const int grp = t / (kGroup * cols);
  const int gsize = min(kGroup, m_tiles - grp * kGroup);
  const int r = t - grp * kGroup * cols;
  const int n = r / gsize;
  PairTile p;
  p.m0 = (grp * kGroup + r - n * gsize) * 256;
  p.n0 = tail ? n_main * bn + n * bn_tail : n * bn;
  p.width = tail ? bn_tail : bn;
  return p;
}

template <int kMode>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmTail, const bf16* __restrict__ bias, const bf16* residual, bf16* y, int M,
                 int N, int K, int epilogue, int m_tiles, int n_main, int bn, int bn_tail, int n_tiles, int stages,
                 const __grid_constant__ RopeArgs rope, int hd) {
  constexpr bool kGated = kMode == kPairGated || kMode == kPairGatedAct;
  extern __shared__ uint8_t smem_raw[];
  // SWIZZLE_128B operands need 1024-byte alignment (the same offset in both CTAs)
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int stage_bytes = kPairABytes + bn * kBlockK;  // bn / 2 weight rows of 128 bytes
  uint8_t* stage_mem = smem + stages * stage_bytes;
  uint8_t* bar_mem = stage_mem + 8 * kPairStageBytes;
  const uint32_t full_bar = smem_addr(bar_mem);                 // leader's: both CTAs' operands of a stage have landed
  const uint32_t empty_bar = full_bar + 8 * kPairMaxStages;     // each CTA's: the stage's MMAs are done
  const uint32_t tfull_bar = empty_bar + 8 * kPairMaxStages;    // each CTA's: an accumulator is complete (2 stages)
  const uint32_t tempty_bar = tfull_bar + 16;                   // leader's: both CTAs' epilogues have read it
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bar_mem + 8 * (2 * kPairMaxStages + 4));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = pair_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int num_kb = K / kBlockK;
  const int num_tiles = m_tiles * n_tiles;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < stages; ++s) {
      mbar_init(full_bar + 8 * s, 1);
      mbar_init(empty_bar + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar + 8 * a, 1);
      mbar_init(tempty_bar + 8 * a, 16);  // one arrive per epilogue warp of the pair
    }
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc_pair(smem_addr(tmem_ptr_smem), 2 * kPairAccCols);
  tcgen05_fence_before();
  pair_barrier();  // the peer's barriers exist before anything arrives there
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;

  if (warp == 0) {
    if (lane == 0) {
      const uint32_t lead_full = pair_map(full_bar, 0);
      auto load_a = [&](const PairTile& t, int kb, int s) {
        tma_load_2d_pair(smem_addr(smem) + s * stage_bytes, &tmA, lead_full + 8 * s, kb * kBlockK, t.m0 + (int)rank * 128);
      };
      // this CTA's half of the tile's weight rows (and the leader announces what both CTAs will load)
      auto load_b = [&](const PairTile& t, int kb, int s) {
        if (rank == 0) mbar_expect_tx(full_bar + 8 * s, 2 * (kPairABytes + t.width * kBlockK));
        int row;
        if (kGated) {  // gate rows in the leader, the up rows that belong to them in the peer
          const int out = t.n0 >> 1;
          row = ((out >> 7) << 8) + (out & 127) + (int)rank * 128;
        } else {
          row = t.n0 + (int)rank * (t.width >> 1);
        }
        tma_load_2d_pair(smem_addr(smem) + s * stage_bytes + kPairABytes, t.width == bn ? &tmB : &tmTail, lead_full + 8 * s,
                         kb * kBlockK, row);
      };
      // weights do not depend on the previous kernel: the first ring of them goes out before the dependency wait
      const int pre = pair < num_tiles ? min(stages, num_kb) : 0;
      const PairTile first = pair_tile(pre ? pair : 0, m_tiles, n_main, bn, bn_tail, n_tiles);
      for (int kb = 0; kb < pre; ++kb) load_b(first, kb, kb);
      pdl_wait();
      pdl_trigger();  // every CTA is resident: the next kernel's may come in as these leave
      for (int kb = 0; kb < pre; ++kb) load_a(first, kb, kb);
      int s = pre == stages ? 0 : pre;
      uint32_t ph = pre == stages ? 0 : 1;  // parity of the empty barrier's phase this lap waits for
      for (int tile = pair; tile < num_tiles; tile += pairs) {
        const PairTile t = pair_tile(tile, m_tiles, n_main, bn, bn_tail, n_tiles);
        for (int kb = tile == pair ? pre : 0; kb < num_kb; ++kb) {
          mbar_wait(empty_bar + 8 * s, ph);
          load_b(t, kb, s);
          load_a(t, kb, s);
          if (++s == stages) s = 0, ph ^= 1;
        }
      }
      // the last arrivals from the leader have come before this CTA may leave
      for (int i = 0; i < stages; ++i) {
        mbar_wait(empty_bar + 8 * s, ph);
        if (++s == stages) s = 0, ph ^= 1;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0) {
      const uint64_t adesc0 = make_smem_desc(smem_addr(smem));
      const uint64_t bdesc0 = make_smem_desc(smem_addr(smem) + kPairABytes);
      int s = 0;
      uint32_t ph = 0, tl = 0;
      for (int tile = pair; tile < num_tiles; tile += pairs, ++tl) {
        const PairTile t = pair_tile(tile, m_tiles, n_main, bn, bn_tail, n_tiles);
        const uint32_t idesc = make_idesc_pair(t.width);
        const uint32_t as = tl & 1;
        mbar_wait(tempty_bar + 8 * as, ((tl >> 1) & 1) ^ 1);  // both epilogues have drained this accumulator
        tcgen05_fence_after();
        const uint32_t tacc = tmem_base + as * kPairAccCols;
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(full_bar + 8 * s, ph);
          tcgen05_fence_after();
          const uint64_t off = (uint64_t)(s * (stage_bytes >> 4));  // start-address field: bytes >> 4
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < kBlockK / kUmmaK; ++k)
              umma_bf16_pair(tacc, adesc0 + off + 2 * k, bdesc0 + off + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            umma_commit_pair(empty_bar + 8 * s, 3);
            if (kb == num_kb - 1) umma_commit_pair(tfull_bar + 8 * as, 3);
          }
          __syncwarp();
          if (++s == stages) s = 0, ph ^= 1;
        }
      }
    }
  } else {
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lead_tempty = pair_map(tempty_bar, 0);
    pdl_wait();  // residual and bias may come from the previous kernel
    uint32_t tl = 0;
    for (int tile = pair; tile < num_tiles; tile += pairs, ++tl) {
      const PairTile t = pair_tile(tile, m_tiles, n_main, bn, bn_tail, n_tiles);
      const uint32_t as = tl & 1;
      const uint32_t lane_base = tmem_base + as * kPairAccCols + ((uint32_t)(quad * 32) << 16);
      int pos = 0;
      size_t cache_row = 0;  // ((page * KV) * page_size + slot): + kvh * page_size gives the token's row of a kv head
      if (kMode == kPairRope && t.m0 + (int)rank * 128 + quad * 32 + lane < M) {
        const int m = t.m0 + (int)rank * 128 + quad * 32 + lane;
        pos = rope.positions[m];
        const int page = rope.page_table[(size_t)rope.seq_ids[m] * rope.max_pages + (pos >> rope.page_shift)];
        cache_row = ((size_t)page * rope.KV << rope.page_shift) + (pos & ((1 << rope.page_shift) - 1));
      }
      // A line of the tile is 64 columns (128 bytes of a row).  The sums leave TMEM with a lane per row, take bias and
      // activation and cross this warp's 4 KB of shared memory as bf16; from there on a lane holds 16 bytes of a row and
      // eight lanes a line of it, so that the residual, the rotation, the cache and y are read and written by whole lines.
      // Straight from the lane that has the row, every 16-byte access of a warp is 32 lines: 5.0 us for the last tile of 224
      // columns, of which nothing hides any.
      uint8_t* const mine = stage_mem + (warp - 2) * kPairStageBytes;
      const auto slot = [&](int row, int chunk) { return reinterpret_cast<uint4*>(mine + row * 128 + ((chunk ^ (row & 7)) << 4)); };
      const int row0 = t.m0 + (int)rank * 128 + quad * 32;
      if constexpr (kMode == kPairRope) {
        // a unit is 32 rotation pairs (i, i + hd / 2) of a head: chunks 0-3 of a staged line are the first elements, 4-7 the
        // second ones
        const int rh = hd >> 1, per_head = rh >> 5;
        // the bias of a unit's columns: lanes 0-15 two first elements each, lanes 16-31 two second ones
        const auto unit_bias = [&](int u) {
          const int col = t.n0 + (u / per_head) * hd + (u % per_head) * 32 + (lane >> 4) * rh + (lane & 15) * 2;
          return (epilogue & DLI_EPI_BIAS) && u < t.width >> 6 && col < N ? pair_bias(bias + col) : 0u;
        };
        uint32_t next_bias = unit_bias(half);
        mbar_wait(tfull_bar + 8 * as, (tl >> 1) & 1);
        tcgen05_fence_after();
#pragma unroll 1
        for (int u = half; u < t.width >> 6; u += 2) {
          const int hh = u / per_head, e0 = (u - hh * per_head) * 32;
          const int head = t.n0 / hd + hh;  // q heads, then k heads, then v heads
          if (head >= rope.H + 2 * rope.KV) break;
          const uint32_t bb = next_bias;
          next_bias = unit_bias(u + 2);
#pragma unroll
          for (int j = 0; j < 4; ++j) {  // 16 columns: j = 0, 1 the first elements, 2, 3 the second ones
            uint32_t r[16];
            const int c0 = (j >> 1) * rh + e0 + (j & 1) * 16;  // column inside the head
            tmem_ld_32x16(lane_base + hh * hd + c0, r);
            tmem_ld_wait();
            float v[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(r[e]);
            if (epilogue & DLI_EPI_BIAS) {
#pragma unroll
              for (int e = 0; e < 16; e += 2) {
                const uint32_t b = __shfl_sync(0xffffffffu, bb, j * 8 + e / 2);
                v[e] += bf_lo(b);
                v[e + 1] += bf_hi(b);
              }
            }
            *slot(lane, j * 2) = pack8(v);
            *slot(lane, j * 2 + 1) = pack8(v + 8);
          }
          __syncwarp();
          const bool turned = rope.cos_t && head < rope.H + rope.KV;
          const int kvh = head - rope.H - (head < rope.H + rope.KV ? 0 : rope.KV);
          bf16* const cache = head < rope.H ? nullptr : head < rope.H + rope.KV ? rope.k_cache : rope.v_cache;
          const int ch = lane & 3;
          uint4 cs[4], sn[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int p = __shfl_sync(0xffffffffu, pos, q * 8 + (lane >> 2));
            cs[q] = sn[q] = make_uint4(0u, 0u, 0u, 0u);
            if (turned) {  // rows past M have position 0
              cs[q] = ld_16B(rope.cos_t + (size_t)p * rh + e0 + ch * 8);
              sn[q] = ld_16B(rope.sin_t + (size_t)p * rh + e0 + ch * 8);
            }
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int row = q * 8 + (lane >> 2);
            uint4 u1 = *slot(row, ch), u2 = *slot(row, ch + 4);
            if (turned) {
              float x1[8], x2[8], c[8], n[8], o1[8], o2[8];
              unpack8(u1, x1);
              unpack8(u2, x2);
              unpack8(cs[q], c);
              unpack8(sn[q], n);
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                float p1 = x1[e] * c[e], q1 = -x2[e] * n[e], p2 = x2[e] * c[e], q2 = x1[e] * n[e];
                round2_bf16(p1, q1);
                round2_bf16(p2, q2);
                o1[e] = p1 + q1;
                o2[e] = p2 + q2;
              }
              u1 = pack8(o1);
              u2 = pack8(o2);
            }
            const unsigned long long crow = __shfl_sync(0xffffffffu, (unsigned long long)cache_row, row);
            if (row0 + row < M) {
              bf16* dst = y + (size_t)(row0 + row) * N + (size_t)head * hd + e0 + ch * 8;
              st_16B(dst, u1);
              st_16B(dst + rh, u2);
              if (cache) {
                bf16* cd = cache + (crow + ((size_t)kvh << rope.page_shift)) * hd + e0 + ch * 8;
                st_16B(cd, u1);
                st_16B(cd + rh, u2);
              }
            }
          }
          __syncwarp();
        }
      } else {
        const int out0 = kGated ? t.n0 >> 1 : t.n0, outs = kGated ? t.width >> 1 : t.width;
        const int n_out = kGated ? N / 2 : N;
        const bool with_res = !kGated && (epilogue & DLI_EPI_RESIDUAL);
        const int ch = lane & 7;
        uint4 res[2][8];  // the residual of this warp's (at most two) lines: rows q * 4 + lane / 8, columns 8 ch of the line
        if (!kGated) {
#pragma unroll
          for (int li = 0; li < 2; ++li)
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const int row = row0 + q * 4 + (lane >> 3), col = half * 64 + li * 128 + ch * 8;
              res[li][q] = with_res && row < M && col < outs && out0 + col < n_out
                               ? ld_16B(residual + (size_t)row * n_out + out0 + col) : make_uint4(0u, 0u, 0u, 0u);
            }
        }
        // the bias of the lines' columns 2 lane and 2 lane + 1 (it may start anywhere)
        uint32_t bb[2] = {0u, 0u};
        if (!kGated && (epilogue & DLI_EPI_BIAS)) {
#pragma unroll
          for (int li = 0; li < 2; ++li) {
            const int col = out0 + half * 64 + li * 128 + lane * 2;
            if (col < N) bb[li] = pair_bias(bias + col);
          }
        }
        mbar_wait(tfull_bar + 8 * as, (tl >> 1) & 1);
        tcgen05_fence_after();
#pragma unroll
        for (int li = 0; li < (kGated ? 1 : 2); ++li) {
          const int cb = half * 64 + li * 128;
          if (cb >= outs) break;
#pragma unroll 1
          for (int ci = 0; ci < 4 && cb + ci * 16 < outs; ci += 2) {  // 32 columns at a time; what lies past `outs` is not used
            uint32_t r[2][16], r2[2][16];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              tmem_ld_32x16(lane_base + cb + (ci + k) * 16, r[k]);
              if (kGated) tmem_ld_32x16(lane_base + outs + cb + (ci + k) * 16, r2[k]);
            }
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              float v[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[k][j]);
              if (kGated) {
                float up[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) { up[j] = __uint_as_float(r2[k][j]); round2_bf16(v[j], up[j]); }
                gated_combine_n(v, up, kMode == kPairGated ? nullptr : reinterpret_cast<const float*>(bias));
              } else {
                if (epilogue & DLI_EPI_BIAS) {
#pragma unroll
                  for (int j = 0; j < 16; j += 2) {
                    const uint32_t b = __shfl_sync(0xffffffffu, bb[li], (ci + k) * 8 + j / 2);
                    v[j] += bf_lo(b);
                    v[j + 1] += bf_hi(b);
                  }
                }
                if (epilogue & DLI_EPI_GELU_NEW) {
#pragma unroll
                  for (int j = 0; j < 16; j += 2) {
                    round2_bf16(v[j], v[j + 1]);
                    v[j] = gelu_of_bf16(v[j]);
                    v[j + 1] = gelu_of_bf16(v[j + 1]);
                  }
                }
              }
              *slot(lane, (ci + k) * 2) = pack8(v);
              *slot(lane, (ci + k) * 2 + 1) = pack8(v + 8);
            }
          }
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int row = q * 4 + (lane >> 3), col = cb + ch * 8;
            if (row0 + row < M && col < outs && out0 + col < n_out) {
              uint4 u = *slot(row, ch);
              if (with_res) {
                float v[8], rr[8];
                unpack8(u, v);
                unpack8(res[li][q], rr);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] += rr[j];
                u = pack8(v);
              }
              st_16B(y + (size_t)(row0 + row) * n_out + out0 + col, u);
            }
          }
          __syncwarp();
        }
      }
      // this warp is done reading the accumulator stage: hand it back to the MMA warp, if a later tile takes it
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0 && tile + 2 * pairs < num_tiles) mbar_arrive_cluster(lead_tempty + 8 * as);
    }
  }
  tcgen05_fence_before();
  pair_barrier<false>();  // the leader's MMAs have read the peer's shared memory, both epilogues their accumulators
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * kPairAccCols);
  }
}

// ---- host side -------------------------------------------------------------------------------------------------------
template <int kMode>
static int launch_pair(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmTail, const void* bias,
                       const void* residual, void* y, int M, int N, int K, int epilogue, const PairShape& sh, int n_tiles,
                       int stages, size_t smem, cudaStream_t s, const RopeArgs& rope, int hd) {
  static PerDeviceOnce once;
  DLI_ONCE_PER_DEVICE(once, dev, DLI_CUDA_CALL(cudaFuncSetAttribute(gemm_pair_kernel<kMode>,
                                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemMax)));
  const int m_tiles = (M + 255) / 256, tiles = m_tiles * n_tiles;
  const int pairs = sm_count_cached() / 2;
  const cudaError_t e = launch_kernel_cluster(gemm_pair_kernel<kMode>, dim3(2 * (tiles < pairs ? tiles : pairs)),
                                              dim3(kPairThreads), smem, s, 2u, tmA, tmB, tmTail, (const bf16*)bias,
                                              (const bf16*)residual, (bf16*)y, M, N, K, epilogue, m_tiles, sh.n_main, sh.bn,
                                              sh.bn_tail, n_tiles, stages, rope, hd);
  if (e != cudaSuccess) return fail(DLI_ERR_CUDA, "gemm_pair_kernel: %s", cudaGetErrorString(e));
  return DLI_OK;
}

// The cut is the cheapest by a model of the kernel's time, fitted to 240 shapes (768 x 768 ... 28672 x 4096, 257 ... 8 192 rows)
// x up to 14 cuts each, B200: a cut it picks is 1.7 % slower than the best one on average.
//   time = (2.5 us (first loads, last epilogue) + what the busiest pair walks)
//          x 1.24 at 10^12 operations and beyond (the power limit), in proportion below
//   a tile = k-blocks x max(0.083 + 0.00091 width, 0.2) us + 0.0097 width us
// The floor of 0.2 us is the latency of a load over the ring.  The tail pays where the last round of full tiles is far from
// full (28672 x 4096 gated at 1 024 rows: 448 tiles of 256 on 74 pairs are 7 rounds, 444 of them and a tail of 64 wide ones
// 6.25: 183 -> 165 us); a cut with one has to win by 1.5 %.
static const int kPairWidths[] = {256, 240, 224, 208, 192, 176, 160, 144, 128, 112, 96, 80, 64};

static double pair_cost(int M, int N, int K, const PairShape& sh, int pairs) {
  const int m_tiles = (M + 255) / 256, rest = N - sh.n_main * sh.bn;
  const long long t1 = (long long)m_tiles * sh.n_main;
  const long long t2 = rest > 0 ? (long long)m_tiles * ((rest + sh.bn_tail - 1) / sh.bn_tail) : 0;
  const auto tile = [&](int w) {
    const double kb = 0.083 + 0.00091 * w;
    return (double)(K / kBlockK) * (kb > 0.2 ? kb : 0.2) + 0.0097 * w;
  };
  const long long a = t1 / pairs, r = t1 % pairs, b = t2 / pairs, q = t2 % pairs;
  double us = (double)a * tile(sh.bn) + (double)(b + (q > 0)) * tile(sh.bn_tail);  // a pair with a full tile less
  if (r > 0) {
    const double v = (double)(a + 1) * tile(sh.bn) + (double)(b + (r + q > pairs)) * tile(sh.bn_tail);
    if (v > us) us = v;
  }
  const double tera = 2e-12 * M * N * K;
  return (us + 2.5) * (1.0 + 0.24 * (tera < 1.0 ? tera : 1.0)) * (m_tiles <= 2 ? 1.03 : 1.0);  // (no neighbour's L2 lines)
}

namespace {
struct PairKey {
  int dev, mode, M, N, K, hd;
  bool operator==(const PairKey& o) const {
    return dev == o.dev && mode == o.mode && M == o.M && N == o.N && K == o.K && hd == o.hd;
  }
};
struct PairPlan { PairShape shape; double us; };
}  // namespace

// a width is a multiple of 16; gate / up pairs: 128 % (width / 2) == 0; rotation: whole heads
static bool pair_width_ok(PairMode mode, int b, int hd) {
  return b >= 16 && b <= 256 && b % 16 == 0 &&
         (mode == kPairGated || mode == kPairGatedAct ? b % 32 == 0 && 128 % (b / 2) == 0 : mode == kPairRope ? b % hd == 0 : true);
}

int plan_gemm_pair(PairMode mode, int M, int N, int K, int hd, PairShape* shape, double* us) {
  static thread_local RecentResults<PairKey, PairPlan, 32> plans;  // pure functions of the sizes and the device
  const int dev = current_device_slot(), pairs = sm_count_cached() / 2;
  if (dev < 0 || pairs <= 0) return DLI_ERR_CUDA;
  const PairKey key{dev, mode, M, N, K, hd};
  const PairPlan* plan = plans.find(key);
  PairPlan made;
  if (plan == nullptr) {
    const int m_tiles = (M + 255) / 256;
    double best = 1e30;
    PairShape pick = {};
    for (int bn : kPairWidths) {
      if (!pair_width_ok(mode, bn, hd)) continue;
      const int cols = (N + bn - 1) / bn;
      const PairShape whole{bn, cols, bn};
      const double t = pair_cost(M, N, K, whole, pairs);
      if (t < best) best = t, pick = whole;
      // as many columns of full tiles as fill whole rounds (all of them, or one fewer), narrow ones after them
      const int rounds = (int)((long long)cols * m_tiles / pairs);
      for (int q = rounds; q > rounds - 2 && q > 0; --q) {
        const int n_main = (int)((long long)q * pairs / m_tiles);
        if (n_main < 1 || n_main >= cols) continue;
        for (int bt : kPairWidths) {
          if (bt >= bn || !pair_width_ok(mode, bt, hd)) continue;
          const PairShape sh{bn, n_main, bt};
          const double v = 1.015 * pair_cost(M, N, K, sh, pairs);
          if (v < best) best = v, pick = sh;
        }
      }
    }
    made = PairPlan{pick, best};
    plans.put(key, made);
    plan = &made;
  }
  *shape = plan->shape;
  *us = plan->us;
  return DLI_OK;
}

int launch_gemm_pair(PairMode mode, const void* x, const void* w, const void* bias, const void* residual, void* y, int M, int N,
                     int K, int epilogue, const PairShape& sh, cudaStream_t s, const RopeArgs& rope, int hd) {
  const int rest = N - sh.n_main * sh.bn;
  const int n_tiles = sh.n_main + (rest > 0 ? (rest + sh.bn_tail - 1) / sh.bn_tail : 0);
  if (!pair_width_ok(mode, sh.bn, hd) || !pair_width_ok(mode, sh.bn_tail, hd) || sh.bn_tail > sh.bn || sh.n_main < 1 ||
      (sh.n_main - 1) * sh.bn >= N || (long long)((M + 255) / 256) * n_tiles > 0x3fffffff)
    return fail(DLI_ERR_INVALID, "gemm_pair: M=%d N=%d K=%d in %d tiles of %d, then %d, does not fit", M, N, K, sh.n_main, sh.bn,
                sh.bn_tail);
  const int stage_bytes = kPairABytes + sh.bn * kBlockK;
  int stages = (kPairSmemMax - kPairSmemFixed) / stage_bytes;
  if (stages > kPairMaxStages) stages = kPairMaxStages;
  const size_t smem = (size_t)stages * stage_bytes + kPairSmemFixed;
  CUtensorMap tmA, tmB, tmTail;
  int rc;
  if ((rc = make_tmap(&tmA, x, M, K, 128)) != DLI_OK) return rc;
  if ((rc = make_tmap(&tmB, w, N, K, sh.bn / 2)) != DLI_OK) return rc;
  if ((rc = make_tmap(&tmTail, w, N, K, sh.bn_tail / 2)) != DLI_OK) return rc;
  const auto launch = mode == kPairGated      ? launch_pair<kPairGated>
                      : mode == kPairGatedAct ? launch_pair<kPairGatedAct>
                      : mode == kPairRope     ? launch_pair<kPairRope>
                                              : launch_pair<kPairPlain>;
  return launch(tmA, tmB, tmTail, bias, residual, y, M, N, K, epilogue, sh, n_tiles, stages, smem, s, rope, hd);
}

}  // namespace dli
