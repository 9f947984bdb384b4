// Argument block shared by the two prefill-attention kernels.
#pragma once

#include "activation.cuh"
#include "common.cuh"

namespace dgpt {

struct FmhaArgs {
  const void* q;
  long long q_bs, q_rs;
  const int* kv_len;
  int kv_len_all;
  void* o;
  long long o_bs, o_rs;
  int o_f32;
  float* lse;
  int B, H, Tq, D, q_offset, causal, dtype;
  int* status;
  int max_ctas;  // at most this many CTAs, looping over the query tiles (0 = as many as fit)
  int two_cta;  // tensor-core path only: the 128-thread kernel with two CTAs per SM instead of the warp-specialised one
  int pingpong;  // tensor-core path only: the kernel with two query tiles per CTA
  // sliding-window form (dgpt_fmha_window); the defaults leave the kernels as dgpt_fmha_prefill uses them
  int window = 0;           // query i sees keys (q_offset + i - window, q_offset + i]; 0 = all of them (causal only)
  float scale = 0.f;        // score scale; 0 = 1 / sqrt(D)
  long long kv_ts = 0;      // elements between consecutive keys of a head; 0 = D
  int kv_heads = 0;         // key/value heads; query head h reads h / (H / kv_heads); 0 = H
  int keep_first = 0;       // with a window: keys j < keep_first are seen from every distance
  const void* hgate = nullptr;  // [B * Tq, H] in dtype: output of head h is multiplied by sigmoid(hgate)
  long long hgate_rs = 0;
  // gate per output element (dgpt_fmha_prefill_gated), exclusive with hgate
  const void* egate = nullptr;  // [B * Tq, H * D] in dtype: o = round(o) * round(sigmoid(egate))
  long long egate_rs = 0;
  // Probabilities as a bf16 pair, high and low part: two-CTAs-per-SM kernel only, for calls whose other route is the warp-level kernel
  // with its probabilities in fp32
  int split_p = 0;
  int any_run = 0;  // the tensor-core kernels may take dense keys of any length, not only whole tiles (impl 0, output not fp32)
};

// What the tensor-core kernels need besides the three tensor maps.
struct TcParams {
  const int* kv_len;
  int kv_len_all;
  const int* page_table;
  int max_pages;
  int page_tokens;
  void* o;
  long long o_bs, o_rs;
  int o_f32;
  float* lse;
  int H, Tq, q_offset, causal;
  float scale_log2;
  int* status;
  int n_qt, n_work;  // query tiles per (batch, head) and work items in all (a capped grid loops over them)
  int d_head;        // head_dim of the tensors in global memory (32 rides on the 64-wide kernels: the TMA boxes are 64 wide
                     // and the columns past the tensor's extent arrive as zeros, so scores and outputs are unchanged)
  int window;        // 0 = no lower bound
  int keep_first;    // keys below this are seen whatever the window
  int kv_div;        // query heads per key/value head
  const void* hgate; // bf16 [B * Tq, H], or NULL
  long long hgate_rs;
  const __nv_bfloat16* egate;  // [B * Tq, H * d_head], or NULL
  long long egate_rs;
  int BH, group_bh;  // two-query-tile kernel: (batch, head) pairs in all, and how many are worked on at a time
};

// Factor that the per-head output gate puts on row `row` (b * Tq + i) of head h.
template <typename T>
__device__ __forceinline__ float head_gate(const void* hgate, long long rs, long long row, int h) {
  if (hgate == nullptr) return 1.f;
  return 1.f / (1.f + expf(-Io<T>::ld(static_cast<const T*>(hgate) + row * rs + h)));
}
// One element through its gate, with the rounding points of a separate pass over the stored output (sigmoid_gate_kernel).
template <typename T>
__device__ __forceinline__ float gated(float o, float g) {
  return Io<T>::round(o) * Io<T>::round(1.f / (1.f + __expf(-g)));
}
// bf16 keeps 8 bits of the sigmoid, so the one-instruction reciprocal (1 ulp of fp32) gives the same rounded value except
// within 2e-7 of a rounding boundary; the full one cost a fifth of the short kernel (425 against 355 us on config 2's shape).
template <>
__device__ __forceinline__ float gated<__nv_bfloat16>(float o, float g) {
  using B = Io<__nv_bfloat16>;
  return B::round(o) * B::round(rcp_fast(1.f + exp_fast(-g)));
}
// N columns (a multiple of 8) of one output row, gated: the stored row never makes a second trip through memory.  (The
// separate pass took 171 us for 131072 x 256 elements and 597 us for 228480 x 512.)
template <int N>
__device__ __forceinline__ void store_gated(__nv_bfloat16* dst, const float* v, float inv, const __nv_bfloat16* gate) {
  uint4 raw[N / 8];  // all loads before the first store, which the compiler could not prove to be elsewhere
#pragma unroll
  for (int i = 0; i < N / 8; ++i) raw[i] = __ldg(reinterpret_cast<const uint4*>(gate) + i);
#pragma unroll
  for (int i = 0; i < N / 8; ++i) {
    float g[8];
    unpack16<__nv_bfloat16>(raw[i], g);
#pragma unroll
    for (int x = 0; x < 8; ++x) g[x] = gated<__nv_bfloat16>(v[8 * i + x] * inv, g[x]);
    st16<__nv_bfloat16>(dst + 8 * i, g, 1.f);
  }
}
// A row's gate of `bytes` on its way to L2 while the row's scores are worked on (loaded cold in the epilogue it is one more miss to memory per item).
__device__ __forceinline__ void prefetch_gate(const __nv_bfloat16* gate, int bytes) {
  const char* p = reinterpret_cast<const char*>(gate);
  for (int i = 0; i < bytes; i += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + i));
}
// First key tile of `tile` keys inside the window of a query at position `first_q` (the query tile's lowest).
__device__ __forceinline__ int window_first_tile(int window, int first_q, int tile) {
  return window > 0 ? max(0, first_q - window + 1) / tile : 0;
}
// Key tiles ahead of that one that hold kept first keys.  A query tile visits the n_window tiles from `tile0` on and then
// tiles [0, n_kept): its j-th tile is tile_of(j).  (The kept ones last: by then the running maximum is settled, and a tile of
// which a few keys are seen seldom moves it.)
__device__ __forceinline__ int kept_tiles(int keep_first, int tile0, int tile) {
  return min(tile0, (keep_first + tile - 1) / tile);
}
template <bool KEPT>
__device__ __forceinline__ int tile_of(int j, int n_window, int tile0) {
  return KEPT && j >= n_window ? j - n_window : tile0 + j;
}

// warp-level kernel (fmha_simt.cu)
int fmha_simt(const FmhaArgs& a, const KvView& kv, cudaStream_t st);

// short sequences with small heads (fmha_mma.cu); `keys`: the most that a query sees
bool fmha_mma_supported(const FmhaArgs& a, const KvView& kv, long long keys);
int fmha_mma(const FmhaArgs& a, const KvView& kv, long long keys, cudaStream_t st);

// tcgen05 / TMEM kernel (fmha_tc.cu)
bool fmha_tc_supported(const FmhaArgs& a, const dgpt_kv_layout& kv);
int fmha_tc(const FmhaArgs& a, const dgpt_kv_layout& kv, cudaStream_t st);
// the same with two query tiles per CTA taking turns on the tensor cores (fmha_pp.cu); `tp` and the maps come from fmha_tc
struct TcMaps;
int fmha_tc_pp_launch(const FmhaArgs& a, const TcMaps& maps, TcParams p, long long kv_span, cudaStream_t st);
// the persistent warp-specialised kernel with one query tile per work item (fmha_ws.cu)
int fmha_tc_ws_launch(const FmhaArgs& a, const TcMaps& maps, TcParams p, long long kv_span, cudaStream_t st);

}  // namespace dgpt
