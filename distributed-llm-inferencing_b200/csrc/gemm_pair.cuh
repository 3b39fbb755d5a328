// Projections of many rows on pairs of SMs (gemm_pair.cu), as the GEMM entry points call them.
#pragma once
#include "gemm_rows.cuh"

namespace dli {

// How the weight rows are cut: n_main tiles of bn, the rest in tiles of bn_tail.
struct PairShape {
  int bn, n_main, bn_tail;
};

// kPairGatedAct: kPairGated with the activation's parameters in `bias` (a kernel of its own: the test for them inside the
// epilogue made it 3 us longer for a tile of 128 outputs).
enum PairMode { kPairPlain = 0, kPairGated = 1, kPairRope = 2, kPairGatedAct = 3 };

// The cut for [M, K] x [N, K]^T and its estimated time in us (the rule stands beside the definition).  hd: kPairRope only.
int plan_gemm_pair(PairMode mode, int M, int N, int K, int hd, PairShape* shape, double* us);

// y = epi(x w^T).  kPairGated: w is the interleaved gate / up matrix, N counts its rows, `bias` is not used; kPairRope:
// N = (H + 2 KV) hd, no residual, no activation.  The caller has checked the arguments: K % 64 == 0, N % 16 == 0 (gated:
// N % 256 == 0), 16-byte pointers.
int launch_gemm_pair(PairMode mode, const void* x, const void* w, const void* bias, const void* residual, void* y, int M, int N,
                     int K, int epilogue, const PairShape& shape, cudaStream_t s, const RopeArgs& rope = RopeArgs{}, int hd = 128);

}  // namespace dli
