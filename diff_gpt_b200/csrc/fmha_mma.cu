// Attention of short sequences with small heads (bf16, head_dim 32 or 64) with the products in registers: mma.sync on fragments, the keys and
// values of a (sequence, head) in shared memory as a whole.
//
// What bounds such heads is not the tensor pipe but the softmax: a 128 x 128 tile of scores is 16384 exponentials, 1024 clocks of the
// SM's exponential units, where its two products are 256 clocks of tcgen05 (head_dim 32).  The tcgen05 kernel spends 4600 clocks on such
// a tile: each of its few softmax warps waits for a commit, a TMEM load, a barrier, one after the other.  Here a warp is on its own from
// its rows' first score to their last output - scores and probabilities never leave its registers - and sixteen of them fill the SM's
// pipes among themselves.
//   A warp takes 16 rows and walks over their keys 32 at a time: four tiles of 16 x 8 scores, exponentials against a running maximum that only
//   moves when it is exceeded by 2^4 (one vote a step; 2^8 left the largest probabilities further from a whole power of two: error against
//   float64 0.00306 instead of 0.00303), probabilities rounded to bf16 as the A operand of the second product.  (32 rows a warp, which
//   read half the fragments, 221 us where 16 take 198: the steps are latency, and 24 warps hide more of it than 16.  The next step's scores
//   issued ahead of a step's exponentials: 242.)
//   SPLIT: each probability as a pair of bf16 numbers, two second products (see fmha_full).
//   CTAs of 8 warps, three an SM (heads of 64: two); blocks of rows are dealt to the warps in snake order, so that under the causal rule short and long rows
//   come together.
// Measured with the gate, us, tcgen05 kernels / this: 256 x 8 heads of 32 x 512 keys 328 / 198 (44 % of the exponential units, 38 % of the tensor
// pipe, 0.56 instructions a clock and scheduler), x 256 133 / 79, x 128 52 / 39; the choice between them is in fmha_simt.cu.
#include "fmha.cuh"
#include "tcgen05.cuh"

namespace dgpt {

constexpr int kMmWarps = 8, kMmThreads = 32 * kMmWarps, kMmKeys = 32;  // keys of a step

struct MmaArgs {
  const __nv_bfloat16* q;
  long long q_bs, q_rs;
  KvView kv;
  const int* kv_len;
  int kv_len_all;
  __nv_bfloat16* o;
  long long o_bs, o_rs;
  const __nv_bfloat16* gate;
  long long gate_rs;
  int H, Tq, q_offset, causal, splits, room;  // room: keys that fit
  float scale_log2;
};

template <int D>
__device__ __forceinline__ uint32_t mm_at(int row, int chunk) {  // byte offset of 8 columns of a row: eight rows side by side do not collide
  return D == 32 ? row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4) : row * 128 + ((chunk ^ (row & 7)) << 4);
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
  asm("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float mm_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int D, bool SPLIT>
__global__ void __launch_bounds__(kMmThreads, D == 32 ? 3 : 2) fmha_mma_kernel(const __grid_constant__ MmaArgs p) {
  constexpr int KS = D / 16, NT = kMmKeys / 8, OT = D / 8, kChunks = D / 8, kRows = 16;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sK = (uint32_t)__cvta_generic_to_shared(smem), sV = sK + (uint32_t)p.room * D * 2;
  const int j = blockIdx.x % p.splits, bh = blockIdx.x / p.splits, h = bh % p.H, b = bh / p.H;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n_blk = (p.Tq + kRows - 1) / kRows, G = p.splits * kMmWarps, me = j * kMmWarps + warp;
  const int klen = min(min(p.kv_len ? p.kv_len[b] : p.kv_len_all, p.kv.page_tokens), p.room);
  // keys that the CTA's last rows see
  int last_blk = 0;
  for (int r = 0; r * G < n_blk; ++r) last_blk = max(last_blk, min(n_blk - 1, (r & 1) ? r * G + G - 1 - j * kMmWarps : r * G + j * kMmWarps + kMmWarps - 1));
  const int need = max(0, p.causal ? min(klen, p.q_offset + min(p.Tq, (last_blk + 1) * kRows)) : klen);
  const int rows = (need + kMmKeys - 1) / kMmKeys * kMmKeys;
  const __nv_bfloat16 *kb = static_cast<const __nv_bfloat16*>(p.kv.k), *vb = static_cast<const __nv_bfloat16*>(p.kv.v);
  // queries and gates of the CTA's rows on their way to L2 under the keys' loads
  for (int i = threadIdx.x; i < n_blk * kRows; i += kMmThreads) {
    const int blk = i / kRows, r = blk / G, in = (r & 1) ? G - 1 - (blk - r * G) : blk - r * G;
    if (in / kMmWarps != j || i >= p.Tq) continue;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p.q + (long long)b * p.q_bs + (long long)i * p.q_rs + h * D));
    if (p.gate) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.gate + ((long long)b * p.Tq + i) * p.gate_rs + h * D));
  }
#pragma unroll 2
  for (int i = threadIdx.x; i < rows * kChunks; i += kMmThreads) {
    const int row = i / kChunks, c = i - row * kChunks;
    long long off = -1;
    if (row < need) off = b * p.kv.page_stride + h * p.kv.head_stride + (long long)row * (p.kv.token_stride ? p.kv.token_stride : D) + c * 8;
    const uint32_t at = mm_at<D>(row, c);
    const int bytes = off >= 0 ? 16 : 0;  // 0: filled with zeros, so that 0 * x stays 0
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sK + at), "l"(kb + (off >= 0 ? off : 0)), "r"(bytes) : "memory");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sV + at), "l"(vb + (off >= 0 ? off : 0)), "r"(bytes) : "memory");
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // this lane's place in a fragment's rows: the swizzle repeats every 8 rows, so it is the same for every step
  uint32_t k_at[KS / 2], v_at[OT / 2];
#pragma unroll
  for (int kk = 0; kk < KS / 2; ++kk) k_at[kk] = mm_at<D>(lane & 7, 4 * kk + (lane >> 3));
#pragma unroll
  for (int n = 0; n < OT / 2; ++n) v_at[n] = mm_at<D>(((lane >> 3) & 1) * 8 + (lane & 7), 2 * n + (lane >> 4));

#pragma unroll 1
  for (int r = 0; r * G < n_blk; ++r) {
    const int blk = (r & 1) ? r * G + G - 1 - me : r * G + me;
    if (blk >= n_blk) continue;
    const int r0 = blk * kRows;
    uint32_t qa[KS][4];
    {
      const __nv_bfloat16* q0 = p.q + (long long)b * p.q_bs + (long long)min(r0 + g, p.Tq - 1) * p.q_rs + h * D + 2 * t;
      const __nv_bfloat16* q1 = p.q + (long long)b * p.q_bs + (long long)min(r0 + g + 8, p.Tq - 1) * p.q_rs + h * D + 2 * t;
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        qa[k][0] = __ldg(reinterpret_cast<const uint32_t*>(q0 + 16 * k));
        qa[k][1] = __ldg(reinterpret_cast<const uint32_t*>(q1 + 16 * k));
        qa[k][2] = __ldg(reinterpret_cast<const uint32_t*>(q0 + 16 * k + 8));
        qa[k][3] = __ldg(reinterpret_cast<const uint32_t*>(q1 + 16 * k + 8));
      }
    }
    float o[OT][4], top[2] = {-INFINITY, -INFINITY}, lsum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int n = 0; n < OT; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    const int end = p.causal ? min(klen, p.q_offset + min(p.Tq, r0 + kRows)) : klen;
#pragma unroll 1
    for (int k0 = 0; k0 < end; k0 += kMmKeys) {
      const uint32_t kk0 = sK + k0 * (D * 2), vk0 = sV + k0 * (D * 2);
      float s[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
        for (int kk = 0; kk < KS / 2; ++kk) {
          uint32_t kf[4];
          ldsm4(kk0 + k_at[kk] + 8 * n * (D * 2), kf);
          mma16816(s[n], qa[2 * kk], kf[0], kf[1]);
          mma16816(s[n], qa[2 * kk + 1], kf[2], kf[3]);
        }
      }
      if (k0 + kMmKeys > klen || (p.causal && k0 + kMmKeys - 1 > p.q_offset + r0)) {
#pragma unroll
        for (int n = 0; n < NT; ++n) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int key = k0 + 8 * n + 2 * t + (e & 1), row = r0 + g + (e >> 1) * 8;
            if (key >= klen || (p.causal && key > p.q_offset + row)) s[n][e] = -INFINITY;
          }
        }
      }
      // exponents against the running maxima; if one exceeds its row's by 2^4 the maxima move (always so at a row's first keys)
      float mx[2], most = -INFINITY;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        mx[e] = fmaxf(s[0][2 * e], s[0][2 * e + 1]);
#pragma unroll
        for (int n = 1; n < NT; ++n) mx[e] = fmaxf(mx[e], fmaxf(s[n][2 * e], s[n][2 * e + 1]));
        most = fmaxf(most, top[e] == -INFINITY ? INFINITY : fmaf(mx[e], p.scale_log2, -top[e]));
      }
      if (__any_sync(0xffffffffu, most > 4.f)) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float m = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 1));
          m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
          const float now = fmaxf(top[e], m * p.scale_log2), alpha = now == -INFINITY ? 1.f : mm_ex2(top[e] - now);
          top[e] = now;
          lsum[2 * e] *= alpha;
          lsum[2 * e + 1] *= alpha;
#pragma unroll
          for (int n = 0; n < OT; ++n) {
            o[n][2 * e] *= alpha;
            o[n][2 * e + 1] *= alpha;
          }
        }
      }
      const uint64_t scale2 = tc::pack2(p.scale_log2, p.scale_log2);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float ref = top[e] == -INFINITY ? 0.f : -top[e];
        const uint64_t ref2 = tc::pack2(ref, ref);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          float x, y;
          tc::unpack2(tc::fma2(tc::pack2(s[n][2 * e], s[n][2 * e + 1]), scale2, ref2), x, y);
          s[n][2 * e] = mm_ex2(x);
          s[n][2 * e + 1] = mm_ex2(y);
        }
      }
#pragma unroll
      for (int kk = 0; kk < NT / 2; ++kk) {
        uint32_t pa[4], pl[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float x = s[2 * kk + (e >> 1)][2 * (e & 1)], y = s[2 * kk + (e >> 1)][2 * (e & 1) + 1];
          pa[e] = pack_bf16(x, y);
          if constexpr (SPLIT) pl[e] = pack_bf16(x - __uint_as_float(pa[e] << 16), y - __uint_as_float(pa[e] & 0xffff0000u));
        }
        // the rows' sums, of what the values are weighed with: a product with ones
        mma16816(lsum, pa, 0x3f803f80u, 0x3f803f80u);
        if constexpr (SPLIT) mma16816(lsum, pl, 0x3f803f80u, 0x3f803f80u);
#pragma unroll
        for (int n = 0; n < OT / 2; ++n) {
          uint32_t vf[4];
          ldsm4t(vk0 + v_at[n] + 16 * kk * (D * 2), vf);
          mma16816(o[2 * n], pa, vf[0], vf[1]);
          mma16816(o[2 * n + 1], pa, vf[2], vf[3]);
          if constexpr (SPLIT) {
            mma16816(o[2 * n], pl, vf[0], vf[1]);
            mma16816(o[2 * n + 1], pl, vf[2], vf[3]);
          }
        }
      }
    }
    // ---- the rows' results: four lanes hold a row in pairs of columns; they swap them so that each has 16 bytes in a run ----
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float sum = lsum[2 * e];  // the same in all four lanes
      const float inv = sum > 0.f ? 1.f / sum : 0.f;
      const int row = r0 + g + 8 * e;
#pragma unroll
      for (int n4 = 0; n4 < OT; n4 += 4) {
        uint32_t v[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) v[n] = pack_bf16(o[n4 + n][2 * e] * inv, o[n4 + n][2 * e + 1] * inv);
        auto pick = [&](int i) { return i == 0 ? v[0] : i == 1 ? v[1] : i == 2 ? v[2] : v[3]; };
        uint32_t w[4];
        const uint32_t a0 = pick(t), a1 = __shfl_xor_sync(0xffffffffu, pick(t ^ 1), 1), a2 = __shfl_xor_sync(0xffffffffu, pick(t ^ 2), 2),
                       a3 = __shfl_xor_sync(0xffffffffu, pick(t ^ 3), 3);  // a_i: from lane t ^ i of the four
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int x = i ^ t;
          w[i] = x == 0 ? a0 : x == 1 ? a1 : x == 2 ? a2 : a3;
        }
        if (row < p.Tq) {
          const int col = h * D + 8 * (n4 + t);
          const uint4 out = make_uint4(w[0], w[1], w[2], w[3]);
          __nv_bfloat16* dst = p.o + (long long)b * p.o_bs + (long long)row * p.o_rs + col;
          if (p.gate) {
            const uint4 graw = __ldg(reinterpret_cast<const uint4*>(p.gate + ((long long)b * p.Tq + row) * p.gate_rs + col));
            float x[8], gv[8];
            unpack16<__nv_bfloat16>(out, x);
            unpack16<__nv_bfloat16>(graw, gv);
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = gated<__nv_bfloat16>(x[i], gv[i]);
            st16<__nv_bfloat16>(dst, x, 1.f);
          } else {
            *reinterpret_cast<uint4*>(dst) = out;
          }
        }
      }
    }
  }
}

// What the kernel covers: whole sequences or portions over dense keys without window, log-sum-exp or fp32 output, `keys` of them at most.
// Not pages: those are the prompts of decode jobs, whose draws follow the rounding of the tcgen05 kernels.  One job's prompts must not change their kernel
// with the number of pairs either, as they may be prefilled by several ranks.
bool fmha_mma_supported(const FmhaArgs& a, const KvView& kv, long long keys) {
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return a.dtype == DGPT_BF16 && (a.D == 32 || a.D == 64) && !a.lse && !a.o_f32 && a.window == 0 && !a.hgate &&
         (a.kv_heads == 0 || a.kv_heads == a.H) && a.max_ctas == 0 && keys >= 1 && keys * a.D * 4 <= 96 * 1024 && al16(a.q) && al16(a.o) &&
         kv.page_table == nullptr && al16(a.egate) && a.egate_rs % 8 == 0 && (kv.token_stride == 0 || kv.token_stride % 8 == 0) && (a.scale == 0.f);
}

template <int D, bool SPLIT>
static int fmha_mma_launch(const MmaArgs& p, unsigned grid, size_t smem, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(fmha_mma_kernel<D, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) {
    set_error("fmha_mma: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    return DGPT_E_CUDA;
  }
  fmha_mma_kernel<D, SPLIT><<<grid, kMmThreads, smem, st>>>(p);
  return launch_status("fmha_mma");
}

int fmha_mma(const FmhaArgs& a, const KvView& kv, long long keys, cudaStream_t st) {
  MmaArgs p;
  p.q = static_cast<const __nv_bfloat16*>(a.q);
  p.q_bs = a.q_bs;
  p.q_rs = a.q_rs;
  p.kv = kv;
  p.kv_len = a.kv_len;
  p.kv_len_all = a.kv_len_all;
  p.o = static_cast<__nv_bfloat16*>(a.o);
  p.o_bs = a.o_bs;
  p.o_rs = a.o_rs;
  p.gate = static_cast<const __nv_bfloat16*>(a.egate);
  p.gate_rs = a.egate_rs;
  p.H = a.H;
  p.Tq = a.Tq;
  p.q_offset = a.q_offset;
  p.causal = a.causal;
  p.scale_log2 = kLog2e / sqrtf((float)a.D);
  p.room = (int)((keys + kMmKeys - 1) / kMmKeys * kMmKeys);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  // one CTA a (sequence, head), or several that share its rows where that leaves room for more CTAs
  const int rows = 16, most = (a.Tq + rows * kMmWarps - 1) / (rows * kMmWarps);
  const long long pairs = (long long)a.B * a.H;
  long long splits = pairs > 0 ? 2ll * sms / pairs : 1;
  p.splits = (int)(splits < 1 ? 1 : splits > most ? most : splits);
  if (pairs * p.splits > 0x7fffffffll) {
    set_error("fmha_mma: too many sequences");
    return DGPT_E_ARG;
  }
  const unsigned grid = (unsigned)(pairs * p.splits);
  const size_t smem = (size_t)p.room * a.D * 4;
  if (a.D == 32) return a.split_p ? fmha_mma_launch<32, true>(p, grid, smem, st) : fmha_mma_launch<32, false>(p, grid, smem, st);
  return a.split_p ? fmha_mma_launch<64, true>(p, grid, smem, st) : fmha_mma_launch<64, false>(p, grid, smem, st);
}

}  // namespace dgpt
