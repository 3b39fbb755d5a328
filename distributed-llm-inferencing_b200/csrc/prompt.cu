// A prompt pass through a shard's layers in one call: the launches of every layer, in order, from native code.
//
// Per layer it enqueues what a caller of the single entry points would: norm, qkv projection (with RoPE and the cache
// append in its epilogue wherever a projection kernel has that form), attention, output projection, norm, feed-forward.
// Short prompts are bound by the host here: a layer of 19 rows takes the GPU ~100 us, one entry point called through
// Python ~11 us, of which the launch itself is 3-4.
#include "gemm_rows.cuh"

namespace dli {

// gemm_tcgen05.cu; *launches grows by the kernels enqueued
int linear_qkv_append(const void* x, const void* w, const void* bias, void* qkv, int M, int K, const RopeArgs& rope, int hd,
                      bool one_kernel, cudaStream_t s, int* launches);

__global__ void __launch_bounds__(256)
prompt_rows_kernel(int32_t* __restrict__ positions, int32_t* __restrict__ seq_ids, int32_t* __restrict__ last_rows, int B,
                   int T, int prefix, int seq0) {
  pdl_wait();
  pdl_trigger();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < B * T) {
    const int b = i / T;
    positions[i] = prefix + i - b * T;
    seq_ids[i] = seq0 + b;
  }
  if (last_rows != nullptr && i < B) last_rows[i] = (i + 1) * T - 1;
}

}  // namespace dli

extern "C" {

int dli_prompt_rows(int32_t* positions, int32_t* seq_ids, int32_t* last_rows, int B, int T, int prefix, int seq0,
                    dli_stream_t stream) {
  using namespace dli;
  DLI_CHECK_ARG(positions && seq_ids, "dli_prompt_rows: null pointer");
  DLI_CHECK_ARG(B >= 0 && T >= 0 && prefix >= 0 && seq0 >= 0 && (long long)B * T <= 0x7fffffffLL - 256,
                "dli_prompt_rows: bad sizes B=%d T=%d prefix=%d seq0=%d", B, T, prefix, seq0);
  if (B == 0 || T == 0) return DLI_OK;
  DLI_LAUNCH("dli_prompt_rows", prompt_rows_kernel, dim3((B * T + 255) / 256), dim3(256), (size_t)0,
             static_cast<cudaStream_t>(stream), positions, seq_ids, last_rows, B, T, prefix, seq0);
  return DLI_OK;
}

int dli_prompt_layers_bf16(const dli_layer_weights* layers, const dli_prompt_pass* pass, int* launches,
                           dli_stream_t stream) {
  using namespace dli;
  DLI_CHECK_ARG(layers && pass && launches, "dli_prompt_layers_bf16: null pointer");
  const dli_prompt_pass& p = *pass;
  DLI_CHECK_ARG(p.h_in && p.h && p.x && p.qkv && p.attn && p.act && p.positions && p.seq_ids && p.page_table && p.page_rows,
                "dli_prompt_layers_bf16: null buffer");
  DLI_CHECK_ARG(p.n_layers >= 0 && p.B >= 0 && p.T >= 0 && p.d > 0 && p.ff > 0 && p.H > 0 && p.KV > 0 && p.H % p.KV == 0 &&
                    (p.hd == 64 || p.hd == 128) && p.prefix >= -1 && p.max_pages > 0 &&
                    (long long)p.B * p.T <= 0x7fffffffLL,
                "dli_prompt_layers_bf16: bad sizes B=%d T=%d d=%d ff=%d H=%d KV=%d hd=%d prefix=%d", p.B, p.T, p.d, p.ff, p.H,
                p.KV, p.hd, p.prefix);
  DLI_CHECK_ARG(p.page_size >= 8 && (p.page_size & (p.page_size - 1)) == 0,
                "dli_prompt_layers_bf16: page_size must be a power of two >= 8 (got %d)", p.page_size);
  DLI_CHECK_ARG((p.cos == nullptr) == (p.sin == nullptr), "dli_prompt_layers_bf16: cos and sin must both be given or both NULL");
  DLI_CHECK_ARG(aligned16(p.qkv) && aligned16(p.cos) && aligned16(p.sin),
                "dli_prompt_layers_bf16: pointers must be 16-byte aligned");
  *launches = 0;
  const int rows = p.B * p.T;
  if (rows == 0) return DLI_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (p.n_layers == 0 && p.h_in != p.h)  // no projection writes the result
    DLI_CUDA_CALL(cudaMemcpyAsync(p.h, p.h_in, (size_t)rows * p.d * sizeof(bf16), cudaMemcpyDeviceToDevice, s));
  RopeArgs ra;
  ra.cos_t = (const bf16*)p.cos;
  ra.sin_t = (const bf16*)p.sin;
  ra.positions = p.positions;
  ra.seq_ids = p.seq_ids;
  ra.page_table = p.page_table;
  ra.max_pages = p.max_pages;
  ra.H = p.H;
  ra.KV = p.KV;
  ra.page_shift = 0;
  while ((1 << ra.page_shift) < p.page_size) ++ra.page_shift;
  const void* res = p.h_in;  // residual source until the first projection has written h
  int rc, n = 0;
#define DLI_STEP(call)                     \
  do {                                     \
    if ((rc = (call)) != DLI_OK) return rc; \
    *launches = ++n;                       \
  } while (0)
  for (int i = 0; i < p.n_layers; ++i) {
    const dli_layer_weights& L = layers[i];
    const bool gpt2 = L.norm1_b != nullptr;  // LayerNorm, plain GELU feed-forward; else RMSNorm, gated SiLU
    DLI_CHECK_ARG(L.norm1 && L.w_qkv && L.w_o && L.norm2 && L.w_ff && L.w_down && L.k_cache && L.v_cache &&
                      gpt2 == (L.norm2_b != nullptr),
                  "dli_prompt_layers_bf16: layer %d lacks weights or caches", i);
    auto norm = [&](const void* src, const void* w, const void* b) {
      return gpt2 ? dli_add_layernorm_bf16(src, nullptr, w, b, nullptr, p.x, rows, p.d, p.eps, stream)
                  : dli_add_rmsnorm_bf16(src, nullptr, w, nullptr, p.x, rows, p.d, p.eps, stream);
    };
    auto linear = [&](const void* x, const void* w, const void* b, const void* r, void* y, int N, int K, int act) {
      return dli_linear_bf16(x, w, b, r, y, rows, N, K, act | (b ? DLI_EPI_BIAS : 0) | (r ? DLI_EPI_RESIDUAL : 0), stream);
    };
    DLI_STEP(norm(res, L.norm1, L.norm1_b));
    ra.k_cache = (bf16*)L.k_cache;
    ra.v_cache = (bf16*)L.v_cache;
    if ((rc = linear_qkv_append(p.x, L.w_qkv, L.b_qkv, p.qkv, rows, p.d, ra, p.hd, !p.split_rope, s, &n)) != DLI_OK) return rc;
    if (p.prefix >= 0)  // a chunk at positions prefix ..: keys and values from the paged cache
      DLI_STEP(dli_attn_prefill_paged_bf16(p.qkv, p.attn, L.k_cache, L.v_cache, p.page_rows, p.max_pages, p.num_pages, p.B,
                                           p.T, p.prefix, p.H, p.KV, p.hd, p.page_size, p.scale, p.window, stream));
    else if (p.tensor_core)
      DLI_STEP(dli_attn_prefill_tc_bf16(p.qkv, p.attn, p.B, p.T, p.H, p.KV, p.hd, p.scale, p.window, stream));
    else
      DLI_STEP(dli_attn_prefill_bf16(p.qkv, p.attn, p.B, p.T, p.H, p.KV, p.hd, p.scale, p.window, stream));
    DLI_STEP(linear(p.attn, L.w_o, L.b_o, res, p.h, p.d, p.H * p.hd, DLI_EPI_NONE));
    res = p.h;
    DLI_STEP(norm(p.h, L.norm2, L.norm2_b));
    if (gpt2) DLI_STEP(linear(p.x, L.w_ff, L.b_ff, nullptr, p.act, p.ff, p.d, DLI_EPI_GELU_NEW));
    else DLI_STEP(dli_linear_gated_silu_bf16(p.x, L.w_ff, p.act, rows, p.ff, p.d, stream));
    DLI_STEP(linear(p.act, L.w_down, L.b_down, p.h, p.h, p.d, p.ff, DLI_EPI_NONE));
  }
#undef DLI_STEP
  *launches = n;
  return DLI_OK;
}

}  // extern "C"
