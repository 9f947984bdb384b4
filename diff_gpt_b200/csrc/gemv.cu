// bf16 linear layers of one or two rows (requests followed token by token): every weight is read once and used once or
// twice, so the tensor cores have nothing to do and what counts is how fast the rows of W come in.
//   A warp takes a pair of W's rows (the two columns of an interleaved gate) and 16-byte pieces of them side by side, eight loads
//   in flight per lane; the activations come from L1.  Where the pairs are too few to fill the GPU the four warps of a
//   CTA share a pair's K.  Sums in fp32; the epilogues and their rounding are those of gemm_tc.cu.
// Measured in us from memory, one row, cuBLAS / the tcgen05 kernel / this: 1024 x 1024 4.8 / 8.3 / 2.3, 5472 x 1024 4.9 / 10 / 4.0, 1024 x 2736
// 8.1 / 16 / 3.4, 2048 x 8192 21 / 40 / 8.0 (4.2 TB/s), 16384 x 1024 8.1 / 13 / 8.0; two rows of the last 8.0 / 13 / 10.3, four of them 13.2.
#include "activation.cuh"
#include "linear.cuh"
#include "sampling.cuh"

namespace dgpt {

struct GemvParams {
  const __nv_bfloat16 *a, *w, *resid;
  __nv_bfloat16* out;
  long long a_rs, w_rs, resid_rs, out_rs;
  int M, N, K;
  float alpha, limit;
};

constexpr int kGvWarps = 4, kGvAhead = 4;  // pieces of each row in flight

template <int MM, int EPI, bool SHARE>
__global__ void __launch_bounds__(32 * kGvWarps) gemv_kernel(const GemvParams p) {
  __shared__ float sums[kGvWarps][2 * MM];
  dep_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pair = SHARE ? blockIdx.x : blockIdx.x * kGvWarps + warp;
  if (!SHARE && 2 * pair >= p.N) {
    dep_wait();  // no CTA ends before the kernel it depends on
    return;
  }
  const int first = SHARE ? warp : 0, step = SHARE ? kGvWarps : 1;  // of the pieces of 256 columns
  const __nv_bfloat16* w0 = p.w + (long long)(2 * pair) * p.w_rs;
  const __nv_bfloat16* w1 = w0 + p.w_rs;
  float acc[2 * MM] = {};
  const int n_pieces = (p.K + 255) / 256;
  // The weights of the first round come from memory into L2 while the kernel before is still at work.  (Into L2 only: should that kernel
  // have written them, the loads behind the wait see it.)
#pragma unroll
  for (int u = 0; u < kGvAhead; ++u) {
    const int k = (first + u * step) * 256 + lane * 8;
    if (k < p.K && (lane & 7) == 0) {  // a line of 128 bytes
      asm volatile("prefetch.global.L2 [%0];" ::"l"(w0 + k));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(w1 + k));
    }
  }
  dep_wait();
  for (int c0 = first; c0 < n_pieces; c0 += step * kGvAhead) {
    uint4 r0[kGvAhead], r1[kGvAhead];
#pragma unroll
    for (int u = 0; u < kGvAhead; ++u) {
      const int k = (c0 + u * step) * 256 + lane * 8;  // K is a multiple of 8
      r0[u] = r1[u] = make_uint4(0u, 0u, 0u, 0u);
      if (k < p.K) {
        r0[u] = __ldg(reinterpret_cast<const uint4*>(w0 + k));
        r1[u] = __ldg(reinterpret_cast<const uint4*>(w1 + k));
      }
    }
#pragma unroll
    for (int u = 0; u < kGvAhead; ++u) {
      const int k = (c0 + u * step) * 256 + lane * 8;
      if (k >= p.K) break;
      float x0[8], x1[8];
      unpack16<__nv_bfloat16>(r0[u], x0);
      unpack16<__nv_bfloat16>(r1[u], x1);
#pragma unroll
      for (int m = 0; m < MM; ++m) {
        if (m >= p.M) break;
        float y[8];
        ld16<__nv_bfloat16>(p.a + (long long)m * p.a_rs + k, y);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          acc[2 * m] = fmaf(x0[i], y[i], acc[2 * m]);
          acc[2 * m + 1] = fmaf(x1[i], y[i], acc[2 * m + 1]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2 * MM; ++i) acc[i] = warp_sum(acc[i]);
  if (SHARE) {
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < 2 * MM; ++i) sums[warp][i] = acc[i];
    }
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (int i = 0; i < 2 * MM; ++i) acc[i] = (sums[0][i] + sums[1][i]) + (sums[2][i] + sums[3][i]);
  }
  if (lane != 0) return;
  using B = Io<__nv_bfloat16>;
#pragma unroll
  for (int m = 0; m < MM; ++m) {
    if (m >= p.M) break;
    float lo = acc[2 * m], hi = acc[2 * m + 1];
    if constexpr (EPI == 1 || EPI == 5) {
      float r;
      if constexpr (EPI == 5) {
        r = silu_mul_fast(lo, hi);
      } else {  // the reference's Linear writes bf16 before the activation reads it
        const float g = fminf(B::round(lo), p.limit);
        const float lin = fminf(fmaxf(B::round(hi), -p.limit), p.limit);
        const float sg = B::round(rcp_fast(1.f + exp_fast(-B::round(p.alpha * g))));
        r = B::round(g * sg) * B::round(lin + 1.f);
      }
      B::st(p.out + (long long)m * p.out_rs + pair, r);
    } else {
      if constexpr (EPI == 2) {
        const __nv_bfloat16* src = p.resid + (long long)m * p.resid_rs + 2 * pair;
        lo += B::ld(src);
        hi += B::ld(src + 1);
      } else if constexpr (EPI == 4) {
        lo = xielu_fast(lo, p.alpha, p.limit);
        hi = xielu_fast(hi, p.alpha, p.limit);
      } else if constexpr (EPI == 6) {
        lo = softcap_logit(B::round(lo), p.alpha);
        hi = softcap_logit(B::round(hi), p.alpha);
      }
      *reinterpret_cast<__nv_bfloat162*>(p.out + (long long)m * p.out_rs + 2 * pair) = __floats2bfloat162_rn(lo, hi);
    }
  }
}

template <int EPI>
static void gemv_run(const GemvParams& p, cudaStream_t st) {
  const int pairs = p.N / 2;
  // sixteen warps on every SM, or the four warps of a CTA on one pair
  const bool share = pairs < 148 * 16 && p.K >= 512;
  const dim3 grid((unsigned)(share ? pairs : (pairs + kGvWarps - 1) / kGvWarps)), block(32 * kGvWarps);
  if (p.M == 1) {
    if (share) launch_few(true, gemv_kernel<1, EPI, true>, grid, block, 0, st, p);
    else launch_few(true, gemv_kernel<1, EPI, false>, grid, block, 0, st, p);
  } else {
    if (share) launch_few(true, gemv_kernel<2, EPI, true>, grid, block, 0, st, p);
    else launch_few(true, gemv_kernel<2, EPI, false>, grid, block, 0, st, p);
  }
}

int gemv_launch(const void* a, int64_t a_row_stride, const void* w, int64_t w_row_stride, void* out, int64_t out_row_stride,
                const void* resid, int64_t resid_row_stride, int32_t M, int32_t N, int32_t K, int32_t epilogue, float alpha, float limit,
                cudaStream_t st) {
  const GemvParams p{static_cast<const __nv_bfloat16*>(a), static_cast<const __nv_bfloat16*>(w), static_cast<const __nv_bfloat16*>(resid),
                     static_cast<__nv_bfloat16*>(out), a_row_stride, w_row_stride, resid_row_stride, out_row_stride, M, N, K, alpha, limit};
  switch (epilogue) {
    case 0: gemv_run<0>(p, st); break;
    case 1: gemv_run<1>(p, st); break;
    case 2: gemv_run<2>(p, st); break;
    case 4: gemv_run<4>(p, st); break;
    case 5: gemv_run<5>(p, st); break;
    default: gemv_run<6>(p, st); break;
  }
  return launch_status("linear");
}

}  // namespace dgpt
