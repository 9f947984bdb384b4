// fp32 linear layers of small models, where a launch's latency and not its arithmetic is the cost (a decode step of the smallest
// reference configuration is nine products of 0.1 to 7 MFLOP):
//   acc[m, n] = sum_k a[m, k] * w[n, k]        a: [M, K], w: nn.Linear weight [N, K], both fp32
//   epilogue 0:  out[m, n]     = acc
//   epilogue 1:  out[m, n / 2] = swiglu(acc[m, n], acc[m, n + 1])   for even n  (the rule of dgpt_swiglu)
//   epilogue 2:  out[m, n]     = resid[m, n] + acc                  (resid may be out)
//   epilogue 6:  out[m, n]     = cap * tanh(acc / cap)
// A CTA of 128 threads makes 16 x 32 outputs, so that 100 rows of 64 columns are still 14 CTAs, each with its whole K (up to 128
// at a time) in shared memory after one round of loads.  Each of its four warps multiplies a quarter of K for the whole tile (4 x 4
// outputs a lane: eight 16-byte reads for 64 multiply-adds) and the quarters are added in shared memory: a chain of K / 16 steps,
// where one warp per quarter of the tile has K / 4 of them.
// Measured in us, cuBLAS -> this: 100 x 256 x 64 3.63 -> 2.62, 100 x 64 x 128 4.65 -> 2.93, 24 x 256 x 512 9.5 -> 7.0, 400 x 256 x 64 3.67 -> 3.26;
// level at about 400 tiles.  With one warp per quarter of the tile 3.39 and 4.40 for the first two.
#include "common.cuh"

namespace dgpt {

constexpr int kLfM = 16, kLfN = 32, kLfK = 128, kLfThreads = 128;
constexpr int kLfPitch = kLfK + 4;  // rows start four banks apart: eight of them read side by side do not collide

struct LinearF32 {
  const float *a, *w, *resid;
  float* out;
  long long a_rs, w_rs, resid_rs, out_rs;
  int M, N, K;
  float alpha, limit;
};

template <int EPI>
__global__ void __launch_bounds__(kLfThreads) linear_f32_kernel(const LinearF32 p) {
  __shared__ __align__(16) float smem[kLfM + kLfN][kLfPitch];
  float(*sa)[kLfPitch] = smem, (*sw)[kLfPitch] = smem + kLfM;
  dep_wait();
  const int tid = threadIdx.x, warp = tid >> 5, ly = (tid & 31) >> 3, lx = tid & 7;
  const int m0 = blockIdx.y * kLfM, n0 = blockIdx.x * kLfN;
  float part[4][4] = {};  // rows ly + 4 i, columns lx + 8 j
  for (int k0 = 0; k0 < p.K; k0 += kLfK) {
    const int vecs = min(kLfK, p.K - k0) >> 2;  // K is a multiple of 4
    if (k0 > 0) __syncthreads();
#pragma unroll
    for (int i = 0; i < (kLfM + kLfN) * (kLfK / 4) / kLfThreads; ++i) {
      const int idx = tid + i * kLfThreads, r = idx / (kLfK / 4), v = idx - r * (kLfK / 4);
      if (v >= vecs) continue;
      const bool is_a = r < kLfM;
      const int row = is_a ? m0 + r : n0 + r - kLfM;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row < (is_a ? p.M : p.N))
        x = *reinterpret_cast<const float4*>((is_a ? p.a + (long long)row * p.a_rs : p.w + (long long)row * p.w_rs) + k0 + 4 * v);
      *reinterpret_cast<float4*>(is_a ? &sa[r][4 * v] : &sw[r - kLfM][4 * v]) = x;
    }
    __syncthreads();
#pragma unroll 2
    for (int v = warp; v < vecs; v += 4) {
      float4 x[4], y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[i] = *reinterpret_cast<const float4*>(&sa[ly + 4 * i][4 * v]);
        y[i] = *reinterpret_cast<const float4*>(&sw[lx + 8 * i][4 * v]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          part[i][j] = fmaf(x[i].x, y[j].x, part[i][j]);
          part[i][j] = fmaf(x[i].y, y[j].y, part[i][j]);
          part[i][j] = fmaf(x[i].z, y[j].z, part[i][j]);
          part[i][j] = fmaf(x[i].w, y[j].w, part[i][j]);
        }
      }
    }
  }
  __syncthreads();  // the operands have been read: their place takes the partial sums [warp][row][column]
  float* sums = &sa[0][0];
  static_assert(4 * kLfM * kLfN <= kLfM * kLfPitch + kLfN * kLfPitch, "partial sums in the operands' place");
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) sums[(warp * kLfM + ly + 4 * i) * kLfN + lx + 8 * j] = part[i][j];
  }
  __syncthreads();
  const int ty = tid >> 3, tx = tid & 7;
  float acc[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int at = ty * kLfN + tx + 8 * j;
    acc[j] = (sums[at] + sums[kLfM * kLfN + at]) + (sums[2 * kLfM * kLfN + at] + sums[3 * kLfM * kLfN + at]);
  }
  const int m = m0 + ty;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = n0 + tx + 8 * j;
    if constexpr (EPI == 1) {
      const float lin_raw = __shfl_xor_sync(0xffffffffu, acc[j], 1);  // the odd column beside an even one
      if ((tx & 1) == 0 && m < p.M && n + 1 < p.N) {
        const float g = fminf(acc[j], p.limit), lin = fminf(fmaxf(lin_raw, -p.limit), p.limit);
        p.out[(long long)m * p.out_rs + (n >> 1)] = g * (1.f / (1.f + __expf(-(p.alpha * g)))) * (lin + 1.f);
      }
    } else if (m < p.M && n < p.N) {
      float r = acc[j];
      if (EPI == 2) r += p.resid[(long long)m * p.resid_rs + n];
      if (EPI == 6) r = p.alpha * tanhf(r / p.alpha);
      p.out[(long long)m * p.out_rs + n] = r;
    }
  }
}

}  // namespace dgpt

using namespace dgpt;

extern "C" int dgpt_linear_f32(const float* a, int64_t a_row_stride, const float* w, int64_t w_row_stride, float* out,
                               int64_t out_row_stride, const float* resid, int64_t resid_row_stride, int32_t M, int32_t N, int32_t K,
                               int32_t epilogue, float alpha, float limit, void* stream) {
  DGPT_REQUIRE(a && w && out, "linear_f32: NULL pointer");
  DGPT_REQUIRE(M >= 0 && N > 0 && K > 0 && M <= 65535 * kLfM, "linear_f32: bad sizes");
  DGPT_REQUIRE(epilogue == 0 || epilogue == 1 || epilogue == 2 || epilogue == 6,
               "linear_f32: epilogue must be 0 (store), 1 (SwiGLU of interleaved pairs), 2 (add) or 6 (soft-cap)");
  DGPT_REQUIRE(epilogue != 2 || resid, "linear_f32: epilogue 2 needs the matrix to add");
  DGPT_REQUIRE(epilogue != 6 || alpha > 0.f, "linear_f32: epilogue 6 needs a positive cap");
  DGPT_REQUIRE(epilogue != 1 || N % 2 == 0, "linear_f32: epilogue 1 needs whole column pairs");
  if (K % 4 != 0 || a_row_stride % 4 != 0 || w_row_stride % 4 != 0 ||
      ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) != 0) {
    set_error("linear_f32: a and w must be 16-byte aligned, K and their row strides multiples of 4");
    return DGPT_E_UNSUPPORTED;
  }
  if (M == 0) return DGPT_OK;
  const LinearF32 p{a, w, resid, out, a_row_stride, w_row_stride, resid_row_stride, out_row_stride, M, N, K, alpha, limit};
  const dim3 grid((unsigned)((N + kLfN - 1) / kLfN), (unsigned)((M + kLfM - 1) / kLfM));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (epilogue == 0) launch_dep(linear_f32_kernel<0>, grid, dim3(kLfThreads), 0, st, p);
  else if (epilogue == 1) launch_dep(linear_f32_kernel<1>, grid, dim3(kLfThreads), 0, st, p);
  else if (epilogue == 2) launch_dep(linear_f32_kernel<2>, grid, dim3(kLfThreads), 0, st, p);
  else launch_dep(linear_f32_kernel<6>, grid, dim3(kLfThreads), 0, st, p);
  return launch_status("linear_f32");
}
