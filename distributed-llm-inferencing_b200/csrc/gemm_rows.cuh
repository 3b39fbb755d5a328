// Projections of a few to some thousand rows (gemm_rows.cu), as the GEMM entry points call them.
#pragma once
#include "tcgen05_utils.cuh"

namespace dli {

// What the epilogue of a qkv projection needs to rotate q and k and to append k and v to the paged cache.
struct RopeArgs {
  const bf16* cos_t;           // [max_pos, hd / 2], or NULL: append only
  const bf16* sin_t;
  const int32_t* positions;    // [M]
  const int32_t* seq_ids;      // [M]
  const int32_t* page_table;   // [n_seqs, max_pages]
  bf16* k_cache;               // [num_pages, KV, page_size, hd]
  bf16* v_cache;
  int max_pages, H, KV, page_shift;
};

// How a projection is cut: `bn` activation rows per tile (a multiple of 16, at most 256), K split over a cluster of
// `splits` CTAs (1..8, at most K / 64), a ring of `stages` operand tiles.  pair: the splits are pairs of CTAs (1..4 of them), all
// rows are one tile (288 or 320, a multiple of 32).
struct RowsShape {
  int bn, splits, stages;
  bool pair;
};

enum RowsMode { kRowsPlain = 0, kRowsGated = 1, kRowsRope = 2 };

// The cut for [M, K] x [N, K]^T and its estimated time in us, on single CTAs and on pairs of them (1e30 us: no such cut); the rules
// stand beside the definitions.
int plan_gemm_rows(int M, int N, int K, bool gated, RowsShape* shape, double* us, RowsShape* pair, double* pair_us);

// y = epi(x w^T).  kRowsGated: w is the interleaved gate / up matrix, N counts its rows, `bias` carries the activation's
// parameters; kRowsRope: N = (H + 2 KV) hd, no residual, no activation.  The caller has checked the arguments:
// K % 64 == 0, N % 16 == 0 (gated: N % 256 == 0), 16-byte pointers.
int launch_gemm_rows(RowsMode mode, const void* x, const void* w, const void* bias, const void* residual, void* y, int M,
                     int N, int K, int epilogue, const RowsShape& shape, cudaStream_t s, const RopeArgs& rope = RopeArgs{},
                     int hd = 128);

}  // namespace dli
