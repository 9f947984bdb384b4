// Prefill / chunk attention, warp-level online-softmax kernel (any dtype, any
// head_dim in {8, 16, 32, 64, 128}), plus the dgpt_fmha_prefill entry
// point that chooses between it and the tcgen05 kernel.
//
// A CTA of 128 threads owns a tile of queries of one (batch, head); K and V tiles
// of 32 keys are staged in shared memory as fp32 and read by every query thread
// as broadcasts.  A query is owned by SPLIT adjacent lanes, each holding D/SPLIT
// elements of q and of the output accumulator in registers.  Scores are produced
// eight keys at a time so that the accumulator is rescaled once per eight keys.  Where that leaves few CTAs, eight lanes share a
// query instead, each with every eighth key, and merge at the end (heads up to 32).
#include "common.cuh"
#include "fmha.cuh"

namespace dgpt {

constexpr int kSimtBN = 32;  // keys per shared-memory tile
constexpr int kSimtKB = 8;   // keys per softmax update

template <typename T, int D, int SPLIT, int KEYS>
__global__ void __launch_bounds__(128)
fmha_simt_kernel(const T* __restrict__ q, long long q_bs, long long q_rs, KvView kv, const int* __restrict__ kv_len,
                 int kv_len_all, void* __restrict__ o, long long o_bs, long long o_rs, int o_f32,
                 float* __restrict__ lse, int H, int Tq, int q_offset, int causal, float scale_log2, int window,
                 int keep_first, int kv_div, const void* __restrict__ hgate, long long hgate_rs,
                 const T* __restrict__ egate, long long egate_rs) {
  static_assert(SPLIT == 1 || KEYS == 1, "a query's lanes share its elements or its keys");
  constexpr int DP = D / SPLIT;               // elements per thread
  constexpr int BM = 128 / (SPLIT * KEYS);    // queries per CTA
  constexpr int VEC = Io<T>::kVec16;
  constexpr int KB = KEYS > 1 ? kSimtBN / KEYS : kSimtKB;  // keys per softmax update
  constexpr int PITCH = KEYS > 1 ? D + 4 : D;  // lanes that read KEYS rows side by side do not collide
  __shared__ __align__(16) float Ks[kSimtBN][PITCH];
  __shared__ __align__(16) float Vs[kSimtBN][PITCH];

  const int b = blockIdx.z, h = blockIdx.y;
  const int q0 = blockIdx.x * BM;
  const int tid = threadIdx.x;
  const int qi = q0 + tid / (SPLIT * KEYS);
  const int part = tid % SPLIT;          // its elements
  const int share = KEYS > 1 ? tid % KEYS : 0;  // its keys: share, share + KEYS, ... of a tile
  const bool q_ok = qi < Tq;
  const int klen = kv_len ? kv_len[b] : kv_len_all;
  int kmax = klen;
  if (causal) kmax = min(klen, q_offset + min(q0 + BM, Tq));
  const int my_last = causal ? q_offset + qi : 0x7fffffff;  // last visible key of this query
  const int my_first = window > 0 ? q_offset + qi - window + 1 : 0;

  float qf[DP], acc[DP];
#pragma unroll
  for (int d = 0; d < DP; ++d) {
    acc[d] = 0.f;
    qf[d] = 0.f;
  }
  if (q_ok) {
    const T* qp = q + (long long)b * q_bs + (long long)qi * q_rs + (long long)h * D + part * DP;
#pragma unroll
    for (int d = 0; d < DP; d += VEC) {
      float t[VEC];
      ld16<T>(qp + d, t);
#pragma unroll
      for (int i = 0; i < VEC; ++i) qf[d + i] = t[i] * scale_log2;
    }
  }
  float m = -INFINITY, l = 0.f;
  const T* kbase = static_cast<const T*>(kv.k);
  const T* vbase = static_cast<const T*>(kv.v);

  const int tile0 = window_first_tile(window, q_offset + q0, kSimtBN), n_window = max(0, (kmax + kSimtBN - 1) / kSimtBN - tile0);
  const int n_tiles = n_window + kept_tiles(keep_first, tile0, kSimtBN);
  for (int tile = 0; tile < n_tiles; ++tile) {
    const int j0 = tile_of<true>(tile, n_window, tile0) * kSimtBN;
    __syncthreads();
    constexpr int VPR = D / VEC;  // 16-byte vectors per key row
    for (int idx = tid; idx < kSimtBN * VPR; idx += 128) {
      const int tk = idx / VPR, pv = idx - tk * VPR;
      const int slot = j0 + tk;
      float kf[VEC], vf[VEC];
      if (slot < klen) {
        const long long off = kv_offset(kv, b, h / kv_div, slot, D) + pv * VEC;
        ld16<T>(kbase + off, kf);
        ld16<T>(vbase + off, vf);
      } else {
#pragma unroll
        for (int i = 0; i < VEC; ++i) kf[i] = vf[i] = 0.f;
      }
#pragma unroll
      for (int i = 0; i < VEC; i += 4) {
        *reinterpret_cast<float4*>(&Ks[tk][pv * VEC + i]) = make_float4(kf[i], kf[i + 1], kf[i + 2], kf[i + 3]);
        *reinterpret_cast<float4*>(&Vs[tk][pv * VEC + i]) = make_float4(vf[i], vf[i + 1], vf[i + 2], vf[i + 3]);
      }
    }
    __syncthreads();
    const int jn = min(kSimtBN, kmax - j0);
    for (int kb = 0; kb < jn; kb += KB * KEYS) {
      float s[KB];
      float smax = -INFINITY;
#pragma unroll
      for (int kk = 0; kk < KB; ++kk) {
        const float* kr = &Ks[kb + kk * KEYS + share][part * DP];
        float dot = 0.f;
#pragma unroll
        for (int d = 0; d < DP; d += 4) {
          const float4 kx = *reinterpret_cast<const float4*>(kr + d);
          dot += qf[d] * kx.x + qf[d + 1] * kx.y + qf[d + 2] * kx.z + qf[d + 3] * kx.w;
        }
#pragma unroll
        for (int x = 1; x < SPLIT; x <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, x);
        const int j = j0 + kb + kk * KEYS + share;
        s[kk] = (q_ok && j < klen && j <= my_last && (j >= my_first || j < keep_first)) ? dot : -INFINITY;
        smax = fmaxf(smax, s[kk]);
      }
      if (smax == -INFINITY) continue;  // nothing visible in this group (no shuffles below)
      const float mn = fmaxf(m, smax);
      const float resc = exp2f(m - mn);
      l *= resc;
#pragma unroll
      for (int d = 0; d < DP; ++d) acc[d] *= resc;
#pragma unroll
      for (int kk = 0; kk < KB; ++kk) {
        const float p = exp2f(s[kk] - mn);
        l += p;
        const float* vr = &Vs[kb + kk * KEYS + share][part * DP];
#pragma unroll
        for (int d = 0; d < DP; d += 4) {
          const float4 vx = *reinterpret_cast<const float4*>(vr + d);
          acc[d] += p * vx.x;
          acc[d + 1] += p * vx.y;
          acc[d + 2] += p * vx.z;
          acc[d + 3] += p * vx.w;
        }
      }
      m = mn;
    }
  }
  if constexpr (KEYS > 1) {  // the shares of a query become one
#pragma unroll
    for (int x = 1; x < KEYS; x <<= 1) {
      const float m2 = __shfl_xor_sync(0xffffffffu, m, x), l2 = __shfl_xor_sync(0xffffffffu, l, x), mn = fmaxf(m, m2);
      const float f = m == -INFINITY ? 0.f : exp2f(m - mn), f2 = m2 == -INFINITY ? 0.f : exp2f(m2 - mn);
      l = l * f + l2 * f2;
#pragma unroll
      for (int d = 0; d < DP; ++d) acc[d] = acc[d] * f + __shfl_xor_sync(0xffffffffu, acc[d], x) * f2;
      m = mn;
    }
    if (share != 0) return;
  }
  if (!q_ok) return;
  float inv = l > 0.f ? 1.f / l : 0.f;
  inv *= head_gate<T>(hgate, hgate_rs, (long long)b * Tq + qi, h);
  const long long oo = (long long)b * o_bs + (long long)qi * o_rs + (long long)h * D + part * DP;
  if (o_f32) {
    float* op = static_cast<float*>(o) + oo;
#pragma unroll
    for (int d = 0; d < DP; ++d) op[d] = acc[d] * inv;
  } else {
    T* op = static_cast<T*>(o) + oo;
    if (egate) {
      // All of the row's gate before the first store, which the compiler cannot prove to be elsewhere: loaded one by one between the
      // stores it took 16.2 us for 4 x 8 heads of 64 x 17 fp32 queries, where a separate pass over the output takes 11.2 in all.
      const T* gp = egate + ((long long)b * Tq + qi) * egate_rs + (long long)h * D + part * DP;
      float g[DP];
      if ((reinterpret_cast<uintptr_t>(gp) & 15) == 0) {
#pragma unroll
        for (int d = 0; d < DP; d += VEC) ld16<T>(gp + d, g + d);
      } else {
#pragma unroll
        for (int d = 0; d < DP; ++d) g[d] = Io<T>::ld(gp + d);
      }
#pragma unroll
      for (int d = 0; d < DP; ++d) g[d] = gated<T>(acc[d] * inv, g[d]);
#pragma unroll
      for (int d = 0; d < DP; ++d) Io<T>::st(op + d, g[d]);
    } else {
#pragma unroll
      for (int d = 0; d < DP; ++d) Io<T>::st(op + d, acc[d] * inv);
    }
  }
  if (lse && part == 0) {
    const int Hn = H;
    lse[((long long)b * Tq + qi) * Hn + h] = l > 0.f ? (m + log2f(l)) * kLn2 : -INFINITY;
  }
}

template <typename T, int D>
static int fmha_simt_launch(const FmhaArgs& a, const KvView& kv, cudaStream_t st) {
  constexpr int SPLIT = D > 64 ? D / 64 : 1;
  constexpr int KEYS = D <= 32 ? 8 : 1;
  const float scale_log2 = a.scale > 0.f ? a.scale * kLog2e : kLog2e / sqrtf((float)D);
#define DGPT_SIMT(SS, KK)                                                                                                     \
  fmha_simt_kernel<T, D, SS, KK><<<dim3((unsigned)((a.Tq + 128 / (SS * KK) - 1) / (128 / (SS * KK))), (unsigned)a.H, (unsigned)a.B), 128, 0, st>>>( \
      static_cast<const T*>(a.q), a.q_bs, a.q_rs, kv, a.kv_len, a.kv_len_all, a.o, a.o_bs, a.o_rs, a.o_f32, a.lse, a.H, a.Tq, a.q_offset, \
      a.causal, scale_log2, a.window, a.window > 0 ? a.keep_first : 0, a.kv_heads > 0 ? a.H / a.kv_heads : 1, a.hgate, a.hgate_rs, \
      static_cast<const T*>(a.egate), a.egate_rs)
  // Eight lanes share a query's keys where one lane per query leaves most SMs without a CTA.  (fp32, us: 100 and 1000
  // queries, 4 heads of 16, 89 keys 10.0 -> 4.4 and 10.6 -> 5.7; 300 x 300, 8 heads of 32, 58 -> 17; 4000 queries, 128 CTAs, 11.3
  // either way.)
  const long long ctas = (long long)a.B * a.H * ((a.Tq + 128 / SPLIT - 1) / (128 / SPLIT));
  // Not in bf16 where the log-sum-exp is asked for too (the prompt a batch of rows shares): the order of its sums would follow the
  // number of rows, and a shard of the batch is to give what the whole gives.
  if (KEYS > 1 && ctas <= 74 && !(sizeof(T) == 2 && a.lse)) DGPT_SIMT(1, KEYS);
  else DGPT_SIMT(SPLIT, 1);
#undef DGPT_SIMT
  return launch_status("fmha_simt");
}

int fmha_simt(const FmhaArgs& a, const KvView& kv, cudaStream_t st) {
#define DGPT_F(TT, DD) return fmha_simt_launch<TT, DD>(a, kv, st)
  if (a.dtype == DGPT_F32) {
    switch (a.D) {
      case 8: DGPT_F(float, 8);
      case 16: DGPT_F(float, 16);
      case 32: DGPT_F(float, 32);
      case 64: DGPT_F(float, 64);
      case 128: DGPT_F(float, 128);
    }
  } else if (a.dtype == DGPT_BF16) {
    switch (a.D) {
      case 8: DGPT_F(__nv_bfloat16, 8);
      case 16: DGPT_F(__nv_bfloat16, 16);
      case 32: DGPT_F(__nv_bfloat16, 32);
      case 64: DGPT_F(__nv_bfloat16, 64);
      case 128: DGPT_F(__nv_bfloat16, 128);
    }
  }
#undef DGPT_F
  set_error("fmha_prefill: dtype %d with head_dim %d is not built", a.dtype, a.D);
  return DGPT_E_UNSUPPORTED;
}

}  // namespace dgpt

using namespace dgpt;

// Every query tile in one round of one CTA per SM.
static bool fmha_one_round(const FmhaArgs& a) {
  static int n_sm[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (n_sm[dev] == 0) cudaDeviceGetAttribute(&n_sm[dev], cudaDevAttrMultiProcessorCount, dev);
  return (long long)a.B * a.H * ((a.Tq + 127) / 128) <= n_sm[dev];
}

// Whether the warp-level kernel applies the output gate itself.  One lane gates a query's whole row there, in fp32 with a full division
// per element, which hundreds of short CTAs cannot hide; a pass of its own takes 1.4 to 2 us more than its launch hides.  Measured in us,
// pass / epilogue: fp32 4 x 8 heads of 64 x 17 11.2 / 13.4, 1 x 4 heads of 128 x 8 7.9 / 10.7, 256 x 8 heads of 32 x 8 18.2 / 24.1, of 16 x 2
// 10.2 / 12.4; but heads of 16, 64 x 12 x 8, 7.9 / 6.9, 1 x 4 x 89 within 0.4 of no gate at all.  bf16 256 x 8 heads of 64 x 2 1.15 times the pass, x 8 level.
static bool simt_own_gate(const FmhaArgs& a) {
  const long long pairs = (long long)a.B * a.H;
  return a.dtype == DGPT_BF16 ? a.Tq >= 8 || pairs <= 512 : a.D <= 16 && pairs <= 1024;
}

// Whether the kernel with its products in registers is ahead of the tcgen05 kernels (us, those / this).  Heads of 32: at every size up to 256 keys
// (1 x 8 x 64 keys 7.3 / 5.3, x 256 8.4 / 7.9; 256 x 8 x 64 53 / 27, x 128 52 / 39) and beyond where pairs of sequence and head are many (16 x 12 x 512
// 37.8 / 33.4, 256 x 8 x 512 328 / 198, but 1 x 8 x 512 10.6 / 11.1, 4 x 8 x 640 12.5 / 15.5).  Keys that are not whole tiles, whose probabilities are
// pairs: always (1 x 8 x 300 13.3 / 8.6, 256 x 8 x 200 163 / 79).  Heads of 64, with two CTAs an SM: only those, up to half a tile and behind the
// first one (256 x 8 x 33 60 / 48, x 64 62 / 59, x 100 67 / 77, x 200 186 / 155, x 300 316 / 250; whole tiles x 256 level, 1 x 8 x 256 9.0 / 11.5).
static bool fmha_prefers_mma(const FmhaArgs& a, long long keys) {
  const long long pairs = (long long)a.B * a.H;
  if (a.D == 32) return a.split_p || keys <= 256 || pairs >= 128;
  return a.split_p && (keys <= 64 || keys > 128);
}

static int fmha_full(const void* q, int64_t q_batch_stride, int64_t q_row_stride, const dgpt_kv_layout* kv, const int32_t* kv_len,
                     int32_t kv_len_all, void* o, int64_t o_batch_stride, int64_t o_row_stride, int32_t o_f32, float* lse,
                     const void* egate, int64_t egate_rs, int32_t B, int32_t H, int32_t Tq, int32_t D, int32_t q_offset,
                     int32_t causal, int32_t dtype, int32_t impl, int32_t max_ctas, int32_t* status, void* stream) {
  DGPT_REQUIRE(q && o, "fmha_prefill: NULL pointer");
  DGPT_REQUIRE(B >= 0 && H > 0 && Tq >= 0 && B <= 65535 && H <= 65535, "fmha_prefill: bad sizes");
  DGPT_REQUIRE(kv_len || kv_len_all >= 0, "fmha_prefill: kv length missing");
  DGPT_REQUIRE(q_row_stride % 8 == 0 && q_batch_stride % 8 == 0 && o_row_stride % 8 == 0 && o_batch_stride % 8 == 0,
               "fmha_prefill: strides must be multiples of 8 elements");
  DGPT_REQUIRE(impl >= 0 && impl <= 4,
               "fmha_prefill: impl must be 0 (auto), 1 (warp-level), 2 (tensor-core, one query tile per CTA), 3 (tensor-core, "
               "two CTAs per SM) or 4 (tensor-core, two query tiles per CTA)");
  if (int e = validate_kv(kv, D)) return e;
  if (B == 0 || Tq == 0) return DGPT_OK;
  FmhaArgs a;
  a.q = q; a.q_bs = q_batch_stride; a.q_rs = q_row_stride;
  a.kv_len = kv_len; a.kv_len_all = kv_len_all;
  a.o = o; a.o_bs = o_batch_stride; a.o_rs = o_row_stride; a.o_f32 = o_f32; a.lse = lse;
  a.B = B; a.H = H; a.Tq = Tq; a.D = D; a.q_offset = q_offset; a.causal = causal; a.dtype = dtype;
  a.status = status;
  a.max_ctas = max_ctas;
  a.egate = egate; a.egate_rs = egate_rs;
  a.pingpong = impl == 4;
  // Dense keys that are not whole tiles: the tensor cores from 24 keys on, heads of 32 from 33 (bf16, us, warp-level / tensor cores: heads of
  // 64 x 24 keys, 4 to 2048 pairs of sequence and head, 9.3 to 82 / 7.3 to 51, of 128 12 to 129 / 8.8 to 62; of 32 x 24 3.6 to 40 / 7.2 to 50,
  // x 40 10 to 64 / 7.1 to 49; 777 keys 90 to 555 / 19 to 27).  An output that is stored in fp32 would show that a probability there has
  // 16 bits: it keeps the warp-level kernel.
  const long long dense_keys = causal ? (long long)Tq + q_offset : kv_len ? (long long)kv->page_tokens : (long long)kv_len_all;
  a.any_run = impl == 0 && !o_f32 && dense_keys >= (D == 32 ? 33 : 24);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const KvView view = make_view(kv);
  const bool tc_ok = fmha_tc_supported(a, *kv);
  // Which tensor-core kernel: the persistent warp-specialised one from 640 keys on (5 to 65 % ahead from 1024; 32 sequences of 768, 12
  // heads of 64, 111 against 115 us) and where one round of its CTAs holds every query tile, so that only the length of a tile's chain
  // counts (8 heads of 64: 4 x 640 tokens 12 against 17 us, 3 x 768, 12 heads, 15 against 20; 128 tokens 7.0 against 7.2); else
  // two smaller CTAs per SM, each done with its item after a few key tiles (256 x 512, 8 heads of 32, 285 against 291 us, 256 x 128 44
  // against 57).
  const long long span = causal ? (long long)Tq + q_offset
                                : (kv_len ? (long long)kv->max_pages * kv->page_tokens : (long long)kv_len_all);
  // The other route of dense keys that are not whole tiles is the warp-level kernel, whose probabilities are fp32: here they keep 16
  // bits as a pair.  Error against float64, rope and norm included, of 4 x 12 heads of 64 x 777 tokens: 0.003236 there, 0.003236 with the
  // pair, 0.0035 with one bf16; the whole layer 337 us there, 66 with the pair (1 x 8 heads x 8191: 3896 and 300; 2 x 16 heads of 128 x 1500:
  // 1669 and 89).
  a.split_p = a.any_run && kv->page_table == nullptr && kv->page_tokens % 128 != 0;
  // (With a log-sum-exp the number of rows is no reason: see fmha_simt_launch.)
  a.two_cta = impl == 3 || a.split_p || (impl == 0 && span < 640 && (lse || !fmha_one_round(a)));
  if (impl >= 2 && !tc_ok) {
    set_error("fmha_prefill: the tensor-core kernel does not cover dtype %d, head_dim %d with this layout", dtype, D);
    return DGPT_E_UNSUPPORTED;
  }
  if (impl == 0 && tc_ok && fmha_prefers_mma(a, span) && fmha_mma_supported(a, view, span)) return fmha_mma(a, view, span, st);
  if (tc_ok && impl != 1) return fmha_tc(a, *kv, st);
  if (egate && !simt_own_gate(a) && (B == 1 || o_batch_stride == (int64_t)Tq * o_row_stride)) {
    a.egate = nullptr;
    if (const int e = fmha_simt(a, view, st)) return e;
    return dgpt_sigmoid_gate(o, o_row_stride, egate, egate_rs, (int64_t)B * Tq, H * D, dtype, stream);
  }
  return fmha_simt(a, view, st);
}

extern "C" int dgpt_fmha_prefill(const void* q, int64_t q_batch_stride, int64_t q_row_stride,
                                 const dgpt_kv_layout* kv, const int32_t* kv_len, int32_t kv_len_all, void* o,
                                 int64_t o_batch_stride, int64_t o_row_stride, int32_t o_f32, float* lse, int32_t B,
                                 int32_t H, int32_t Tq, int32_t D, int32_t q_offset, int32_t causal, int32_t dtype,
                                 int32_t impl, int32_t max_ctas, int32_t* status, void* stream) {
  return fmha_full(q, q_batch_stride, q_row_stride, kv, kv_len, kv_len_all, o, o_batch_stride, o_row_stride, o_f32, lse, nullptr, 0, B, H,
                   Tq, D, q_offset, causal, dtype, impl, max_ctas, status, stream);
}

extern "C" int dgpt_fmha_prefill_gated(const void* q, int64_t q_batch_stride, int64_t q_row_stride, const dgpt_kv_layout* kv,
                                       const int32_t* kv_len, int32_t kv_len_all, void* o, int64_t o_batch_stride,
                                       int64_t o_row_stride, const void* gate, int64_t gate_row_stride, int32_t B, int32_t H,
                                       int32_t Tq, int32_t D, int32_t q_offset, int32_t causal, int32_t dtype, int32_t impl,
                                       int32_t* status, void* stream) {
  DGPT_REQUIRE(gate, "fmha_prefill_gated: NULL pointer");
  return fmha_full(q, q_batch_stride, q_row_stride, kv, kv_len, kv_len_all, o, o_batch_stride, o_row_stride, 0, nullptr, gate,
                   gate_row_stride, B, H, Tq, D, q_offset, causal, dtype, impl, 0, status, stream);
}

// Sliding-window attention for both entry points: `kv` with keys kv_ts elements apart, dense runs or pages.
static int fmha_sliding(const char* what, const void* q, int64_t q_batch_stride, int64_t q_row_stride, const dgpt_kv_layout& kv,
                        int64_t kv_ts, int32_t n_keys, void* o, int64_t o_batch_stride, int64_t o_row_stride, const void* gate,
                        int64_t gate_row_stride, int32_t B, int32_t H, int32_t G, int32_t Tq, int32_t D, int32_t q_offset,
                        int32_t window, int32_t keep_first, float scale, int32_t dtype, int32_t impl, int32_t* status, void* stream) {
  DGPT_REQUIRE(q && o, "%s: NULL pointer", what);
  DGPT_REQUIRE(B >= 0 && H > 0 && G > 0 && H % G == 0 && Tq >= 0 && B <= 65535 && H <= 65535 && n_keys >= 0, "%s: bad sizes", what);
  DGPT_REQUIRE(window >= 0 && keep_first >= 0 && q_offset >= 0 && scale > 0.f, "%s: bad window, kept keys, offset or scale", what);
  DGPT_REQUIRE(q_row_stride % 8 == 0 && q_batch_stride % 8 == 0 && o_row_stride % 8 == 0 && o_batch_stride % 8 == 0 && kv_ts > 0 &&
                   kv_ts % 8 == 0,
               "%s: strides must be multiples of 8 elements", what);
  DGPT_REQUIRE(impl >= 0 && impl <= 3, "%s: impl must be 0 (auto), 1 (warp-level), 2 or 3 (tensor-core)", what);
  if (B == 0 || Tq == 0) return DGPT_OK;
  if (int e = validate_kv(&kv, D)) return e;
  DGPT_REQUIRE(n_keys <= (kv.page_table ? (long long)kv.max_pages * kv.page_tokens : (long long)kv.page_tokens),
               "%s: more keys than the layout holds", what);
  FmhaArgs a;
  a.q = q; a.q_bs = q_batch_stride; a.q_rs = q_row_stride;
  a.kv_len = nullptr; a.kv_len_all = n_keys;
  a.o = o; a.o_bs = o_batch_stride; a.o_rs = o_row_stride; a.o_f32 = 0; a.lse = nullptr;
  a.B = B; a.H = H; a.Tq = Tq; a.D = D; a.q_offset = q_offset; a.causal = 1; a.dtype = dtype;
  a.status = status;
  a.max_ctas = 0;
  a.pingpong = 0;
  a.window = window; a.scale = scale; a.kv_ts = kv_ts;
  a.kv_heads = G; a.keep_first = keep_first;
  a.hgate = gate; a.hgate_rs = gate_row_stride;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // The persistent kernel as for full attention, unless the window leaves a query tile only a few key tiles (16 heads, 8192
  // tokens: window 128 39 against 46 us, 512 level, 1024 126 against 107 us).  With kept first keys it is ahead from 512 keys on (256
  // sequences, 16 heads of 128, 776 against 883 us; 8 x 2048, window 512, 143 against 156).
  const bool short_keys = n_keys < (keep_first > 0 ? 512 : 640) && !fmha_one_round(a);
  a.two_cta = impl == 3 || (impl == 0 && (short_keys || (window > 0 && window <= 512 && keep_first == 0)));
  const bool tc_ok = fmha_tc_supported(a, kv);
  if (impl >= 2 && !tc_ok) {
    set_error("%s: the tensor-core kernels do not cover dtype %d, head_dim %d with this layout", what, dtype, D);
    return DGPT_E_UNSUPPORTED;
  }
  if (tc_ok && impl != 1) return fmha_tc(a, kv, st);
  KvView view = make_view(&kv);
  view.token_stride = kv_ts;
  return fmha_simt(a, view, st);
}

extern "C" int dgpt_fmha_window(const void* q, int64_t q_batch_stride, int64_t q_row_stride, const void* k, const void* v,
                                int64_t kv_batch_stride, int64_t kv_row_stride, int64_t kv_head_stride, int32_t n_keys, void* o,
                                int64_t o_batch_stride, int64_t o_row_stride, const void* gate, int64_t gate_row_stride,
                                int32_t B, int32_t H, int32_t Tq, int32_t D, int32_t q_offset, int32_t window, float scale,
                                int32_t dtype, int32_t impl, int32_t* status, void* stream) {
  DGPT_REQUIRE(kv_batch_stride % 8 == 0 && kv_head_stride % 8 == 0, "fmha_window: strides must be multiples of 8 elements");
  dgpt_kv_layout kv = {};
  kv.k_base = const_cast<void*>(k);
  kv.v_base = const_cast<void*>(v);
  kv.page_stride = kv_batch_stride;
  kv.head_stride = kv_head_stride;
  kv.page_tokens = n_keys > 0 ? n_keys : 1;
  return fmha_sliding("fmha_window", q, q_batch_stride, q_row_stride, kv, kv_row_stride, n_keys, o, o_batch_stride, o_row_stride, gate,
                      gate_row_stride, B, H, H, Tq, D, q_offset, window, 0, scale, dtype, impl, status, stream);
}

extern "C" int dgpt_fmha_grouped(const void* q, int64_t q_batch_stride, int64_t q_row_stride, const dgpt_kv_layout* kv,
                                 int64_t kv_token_stride, int32_t n_keys, void* o, int64_t o_batch_stride, int64_t o_row_stride,
                                 int32_t B, int32_t H, int32_t G, int32_t Tq, int32_t D, int32_t q_offset, int32_t window,
                                 int32_t keep_first, float scale, int32_t dtype, int32_t impl, int32_t* status, void* stream) {
  DGPT_REQUIRE(kv, "fmha_grouped: NULL pointer");
  return fmha_sliding("fmha_grouped", q, q_batch_stride, q_row_stride, *kv, kv_token_stride, n_keys, o, o_batch_stride, o_row_stride,
                      nullptr, 0, B, H, G, Tq, D, q_offset, window, keep_first, scale, dtype, impl, status, stream);
}
