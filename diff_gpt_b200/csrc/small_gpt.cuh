// The kernel of small_gpt.cu, in a header so that its widths can be compiled side by side.
#pragma once

#include "sample_row.cuh"
#include "tcgen05.cuh"

namespace dgpt {

constexpr int kSgThreads = 256, kSgWarps = kSgThreads / 32;  // and one more warp, which loads
constexpr int kSgMaxLayers = 16;
constexpr int kSgChunk = 4096;  // floats of a ring slot: 16 KB of weights
constexpr int kSgMaxSlots = 16;
constexpr int kSgGroup = 4;  // chunks between two of the loader's turns: the ring has more slots than that
struct SmallGpt {
  const float *emb, *w, *cs;
  long long n_w;           // floats of the matrices in front of the mix vectors
  KvView kv;               // layer 0
  long long layer_stride;  // elements from one layer's K (V) to the next one's
  const int *ids, *pos0, *slot0, *step, *len0, *start1, *len1;
  float* logits;
  int* status;
  int L, H, V, layers_per_block, table_len;
  int R;               // rows (decode) or sequences (chunk)
  int T, t_base, T_all;  // chunk: tokens of this launch, those before it, those of the call (0 = decode)
  int cluster, last_only, n_steps;
  int slots;               // of the ring
  int max_keys;            // that a row sees
  float alpha, limit, logit_cap;
  // the draw (out_tok NULL: none)
  float cap, temperature, top_p;
  uint32_t seed_lo, seed_hi;
  int log2c, force_rows;
  const long long* traj;
  const int* force;
  long long force_stride, hist_stride;
  int *out_tok, *hist;
};

__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// threadIdx.x read anew: what is computed from it stays in the phase that uses it.  (Hoisted out of the layers' loop, the addresses of all
// phases together fill the registers.)
__device__ __forceinline__ int tid_here() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// The barrier of the warps that compute.
__device__ __forceinline__ void sg_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kSgThreads) : "memory"); }

// The same, telling every thread whether any of them said yes.
__device__ __forceinline__ bool sg_any(bool mine) {
  int r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbarrier.red.or.pred q, 1, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
               : "=r"(r)
               : "r"((int)mine), "n"(kSgThreads)
               : "memory");
  return r != 0;
}

// One product of the CTA's M rows: out[m][n] = sum_k a[m][k] w[n][k], w as [K / 4 / KS][N][KS][4] in kChunks slots of the ring: KS lanes
// side by side share a column, so that a warp reads 512 bytes in a row.  (As [K / 4][N][4] its lanes meet in the same banks, KS deep: the
// 64 x 128 product of one row took 3000 clocks.)
template <int K, int N, int M>
struct Product {
  static constexpr int kWords = K / 4 * N;  // of 16 bytes
  static constexpr int kChunkWords = kWords < kSgChunk / 4 ? kWords : kSgChunk / 4, kChunks = kWords / kChunkWords;
  static constexpr int kRows = kChunkWords / N;  // k words a chunk holds for every column
  static constexpr int kCols = N > kSgThreads ? N / kSgThreads : 1;  // columns of a thread
  static constexpr int KS0 = N > kSgThreads ? 1 : kSgThreads / N, KS = KS0 < kRows ? KS0 : kRows;  // lanes that share a column
  static_assert(kWords % kChunkWords == 0 && kChunkWords % N == 0 && N * KS <= kSgThreads * kCols && KS <= 16 && kRows % KS == 0, "shape");
  static_assert(kChunks <= kSgGroup || kChunks % kSgGroup == 0, "groups");

  // f(m, n, value) for every output; the KS lanes of a column hold the same value, `mine` says which of them should use it.
  // The caller tells the loader that the last group has been read, behind a barrier of its own.
  static constexpr int kGroup = kChunks < kSgGroup ? kChunks : kSgGroup;
  template <typename R, typename F>
  static __device__ __forceinline__ void run(R& ring, const float* a, F&& f) {
    const int tid = tid_here(), n = tid / KS, ks = tid % KS;
    float4 acc[kCols][M];
#pragma unroll
    for (int q = 0; q < kCols; ++q) {
#pragma unroll
      for (int m = 0; m < M; ++m) acc[q][m] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    constexpr bool kAll = N * KS == kSgThreads * kCols;
#pragma unroll 1
    for (int c0 = 0; c0 < kChunks; c0 += kGroup) {
      if (kChunks > kGroup && c0 > 0) {
        sg_sync();
        ring.release(kGroup);
      }
      ring.await(kGroup);
      const float4* w[kGroup];
#pragma unroll
      for (int c = 0; c < kGroup; ++c) w[c] = reinterpret_cast<const float4*>(ring.next()) + tid;
      if (!kAll && tid >= N * KS) continue;
      const float* x0 = a + 4 * (c0 * kRows + ks);
#pragma unroll
      for (int c = 0; c < kGroup; ++c) {
#pragma unroll
        for (int i = 0; i < kRows / KS; ++i) {
          float4 use[kCols];
#pragma unroll
          for (int q = 0; q < kCols; ++q) use[q] = w[c][i * KS * N + q * kSgThreads];
#pragma unroll
          for (int m = 0; m < M; ++m) {
            const float4 x = *reinterpret_cast<const float4*>(x0 + m * K + 4 * (c * kRows + i * KS));
#pragma unroll
            for (int q = 0; q < kCols; ++q) {
              acc[q][m].x = fmaf(x.x, use[q].x, acc[q][m].x);
              acc[q][m].y = fmaf(x.y, use[q].y, acc[q][m].y);
              acc[q][m].z = fmaf(x.z, use[q].z, acc[q][m].z);
              acc[q][m].w = fmaf(x.w, use[q].w, acc[q][m].w);
            }
          }
        }
      }
    }
    if (!kAll && tid >= N * KS) return;
#pragma unroll
    for (int q = 0; q < kCols; ++q) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float s = (acc[q][m].x + acc[q][m].y) + (acc[q][m].z + acc[q][m].w);
#pragma unroll
        for (int o = 1; o < KS; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        f(m, n + q * kSgThreads, s, m % KS == ks);
      }
    }
  }
};

// Depth mix and norm of one row by one warp: candidates `mask` (bit j: cand[j]), candidate 0 counted `mult0` times.
template <int C, int M>
__device__ __forceinline__ void mix_row(const float* cand, int m, unsigned mask, int mult0, const float* w, float* u) {
  constexpr int E = C / 32, U = C == 128 ? 2 : 4;
  const int lane = tid_here() & 31;
  float acc[E] = {}, top = -INFINITY, l = 0.f;
  if ((mask & (mask - 1)) == 0) {  // one candidate: the mix is the identity
    const float* src = cand + ((__ffs(mask) - 1) * M + m) * C;
#pragma unroll
    for (int i = 0; i < E; ++i) acc[i] = src[lane + 32 * i];
    l = 1.f;
  } else {
    float wv[E];
#pragma unroll
    for (int i = 0; i < E; ++i) wv[i] = w[lane + 32 * i];
    for (unsigned left = mask; left;) {  // up to four candidates at a time: their reductions overlap
      float v[U][E], ss[U], dot[U];
      bool there[U];
      int j = 0;
      const bool has0 = left & 1u;
#pragma unroll
      for (int c = 0; c < U; ++c) {
        there[c] = left != 0;
        if (there[c]) j = __ffs(left) - 1;
        left &= left - 1;
        ss[c] = dot[c] = 0.f;
#pragma unroll
        for (int i = 0; i < E; ++i) {
          v[c][i] = cand[(j * M + m) * C + lane + 32 * i];
          ss[c] = fmaf(v[c][i], v[c][i], ss[c]);
          dot[c] = fmaf(v[c][i], wv[i], dot[c]);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int c = 0; c < U; ++c) {
          ss[c] += __shfl_xor_sync(0xffffffffu, ss[c], o);
          dot[c] += __shfl_xor_sync(0xffffffffu, dot[c], o);
        }
      }
      float nt = top;
#pragma unroll
      for (int c = 0; c < U; ++c) {
        dot[c] = there[c] ? dot[c] * rsqrtf(ss[c] / (float)C + kRmsEps) : -INFINITY;
        nt = fmaxf(nt, dot[c]);
      }
      const float resc = __expf(top - nt);
      l *= resc;
#pragma unroll
      for (int i = 0; i < E; ++i) acc[i] *= resc;
#pragma unroll
      for (int c = 0; c < U; ++c) {
        if (!there[c]) continue;
        const float p = __expf(dot[c] - nt) * (c == 0 && has0 ? (float)mult0 : 1.f);
        l += p;
#pragma unroll
        for (int i = 0; i < E; ++i) acc[i] = fmaf(p, v[c][i], acc[i]);
      }
      top = nt;
    }
  }
  const float invl = __fdividef(1.f, l);
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < E; ++i) {
    acc[i] *= invl;
    ss = fmaf(acc[i], acc[i], ss);
  }
  ss = warp_sum(ss);
  const float inv = rsqrtf(ss / (float)C + kRmsEps);
#pragma unroll
  for (int i = 0; i < E; ++i) u[m * C + lane + 32 * i] = acc[i] * inv;
}

constexpr unsigned kNoKey = 0xffffffffu;

// A warp's round of keys: D / 4 lanes read a key together, so that a load is whole lines (a lane per key touches sixteen lines with every
// load: 4400 clocks for 137 keys of 4 heads), four such loads of K and of V in flight.  Key `fresh` lies in shared memory, at kn and vn
// (generic loads serve both).
template <int D>
struct KeyRound {
  static constexpr int kLanes = D / 4, G = 32 / kLanes, U = 4;
  float4 k[U], v[U];
  unsigned ok;

  // `at`: where key i begins in units of 16 bytes (kNoKey: nowhere), `n` of them
  __device__ __forceinline__ void load(const unsigned* at, int n, const float* kb, const float* vb, const float* kn, const float* vn, int fresh,
                                       int j0) {
    const int lane = tid_here() & 31, g = lane / kLanes, e = lane % kLanes;
    ok = 0u;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = j0 + u * G + g;
      const unsigned off = i < n ? at[i] : kNoKey;
      const bool in = off != kNoKey;
      const float4* kp = reinterpret_cast<const float4*>(i == fresh ? kn : kb + 4ull * off) + e;
      const float4* vp = reinterpret_cast<const float4*>(i == fresh ? vn : vb + 4ull * off) + e;
      k[u] = v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (in) {
        ok |= 1u << u;
        k[u] = *kp;
        v[u] = *vp;
      }
    }
  }
};

// Attention of one (row, head) over this warp's share of the keys, the first round of which is in `r`; the next one is on its way
// while one is worked on.  Every group of lanes has a softmax of its own; they are merged once, at the end.  out: D sums, maximum (log2
// domain), sum of exponentials.
template <int D>
__device__ __forceinline__ void attend(const unsigned* at, int n, const float* kb, const float* vb, KeyRound<D>& r, const float* q, const float* kn,
                                       const float* vn, int fresh, int part, int parts, float* out) {
  constexpr int kLanes = KeyRound<D>::kLanes, G = KeyRound<D>::G, U = KeyRound<D>::U;
  const int lane = tid_here() & 31, g = lane / kLanes, e = lane % kLanes;
  const float4 x = *reinterpret_cast<const float4*>(q + 4 * e);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float top = -INFINITY, l = 0.f;
#pragma unroll 1
  for (int j0 = part * G * U;;) {
    KeyRound<D> now = r;
    if (fresh >= j0 && fresh < j0 + G * U) {  // made after the round was loaded
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (j0 + u * G + g == fresh) {
          now.k[u] = *reinterpret_cast<const float4*>(kn + 4 * e);
          now.v[u] = *reinterpret_cast<const float4*>(vn + 4 * e);
        }
      }
    }
    j0 += parts * G * U;
    const bool more = j0 < n;
    if (more) r.load(at, n, kb, vb, kn, vn, fresh, j0);
    float sc[U], nt = top;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      sc[u] = fmaf(x.x, now.k[u].x, x.z * now.k[u].z) + fmaf(x.y, now.k[u].y, x.w * now.k[u].w);
#pragma unroll
      for (int o = 1; o < kLanes; o <<= 1) sc[u] += __shfl_xor_sync(0xffffffffu, sc[u], o);
      if (!(now.ok >> u & 1u)) sc[u] = -INFINITY;
      nt = fmaxf(nt, sc[u]);
    }
    const float ref = nt == -INFINITY ? 0.f : nt, resc = exp2_fast(top - ref);
    l *= resc;
    acc.x *= resc; acc.y *= resc; acc.z *= resc; acc.w *= resc;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float p = exp2_fast(sc[u] - ref);
      l += p;
      acc.x = fmaf(p, now.v[u].x, acc.x);
      acc.y = fmaf(p, now.v[u].y, acc.y);
      acc.z = fmaf(p, now.v[u].z, acc.z);
      acc.w = fmaf(p, now.v[u].w, acc.w);
    }
    top = nt;
    if (!more) break;  // the same for every lane
  }
  float all = top;
#pragma unroll
  for (int o = kLanes; o < 32; o <<= 1) all = fmaxf(all, __shfl_xor_sync(0xffffffffu, all, o));
  const float f = all == -INFINITY ? 0.f : exp2_fast(top - all);
  l *= f;
  acc.x *= f; acc.y *= f; acc.z *= f; acc.w *= f;
#pragma unroll
  for (int o = kLanes; o < 32; o <<= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, o);
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
    acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
  }
  if (g == 0) *reinterpret_cast<float4*>(out + 4 * e) = acc;
  if (lane == 0) *reinterpret_cast<float2*>(out + D) = make_float2(all, l);
}

// The draw of sample_row where nothing is filtered and a lane's run of tokens fits its registers (CH a lane, V <= 32 CH): the same sums in
// the same order, without a trip through shared memory per token.  `bits`: the random word of (trajectory, step).
template <int CH>
__device__ __forceinline__ int draw_row(const float* z, int V, float temperature, uint32_t bits) {
  const int lane = tid_here() & 31, c0 = lane * CH;
  float e[CH];
  ArgMax best{-INFINITY, 0x7fffffff};
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    e[i] = c0 + i < V ? z[c0 + i] : -INFINITY;
    if (e[i] > best.v) best = ArgMax{e[i], c0 + i};
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax t;
    t.v = __shfl_xor_sync(0xffffffffu, best.v, o);
    t.i = __shfl_xor_sync(0xffffffffu, best.i, o);
    best = better(best, t);
  }
  if (temperature == 0.f) return best.i;
  float mine = 0.f;
#pragma unroll
  for (int i = 0; i < CH; ++i) e[i] = c0 + i < V ? __expf(e[i] - best.v) : 0.f;
  if (temperature != 1.f) {
    const float inv_t = 1.f / temperature;
#pragma unroll
    for (int i = 0; i < CH; ++i) e[i] = e[i] == 0.f ? 0.f : __expf(__logf(e[i]) * inv_t);
  }
#pragma unroll
  for (int i = 0; i < CH; ++i) mine += e[i];
  float incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const float W = __shfl_sync(0xffffffffu, incl, 31), tgt = (float)(bits >> 8) * (1.0f / 16777216.0f) * W;
  float local, c = 0.f;
  const int who = walk_owner(mine, incl, tgt, &local);
  int pick = best.i;
  bool on = true;
#pragma unroll
  for (int i = 0; i < CH; ++i) {  // every lane walks its own run; the owner's result counts
    c += e[i];
    if (on && e[i] > 0.f) pick = c0 + i;
    on = on && !(e[i] > 0.f && c > local);
  }
  return who < 0 ? best.i : __shfl_sync(0xffffffffu, pick, who);  // no sum to walk along, as sample_row
}

// What the ring receives, in the order of use: per layer the four matrices, then the head's blocks of 256 columns, and again.
template <int C>
struct SgChunks {
  static constexpr int kQ = Product<C, 4 * C, 1>::kChunks, kP = Product<C, C, 1>::kChunks, kD = Product<2 * C, C, 1>::kChunks;
  static constexpr int kLayer = 2 * kQ + kP + kD, kHead = Product<C, 256, 1>::kChunks;
  static __device__ __forceinline__ int floats(int in_layer) {  // of a layer's chunk
    if (C >= 64) return kSgChunk;
    return in_layer == kQ ? C * C : in_layer == 2 * kQ + kP ? 2 * C * C : kSgChunk;
  }
};

// The reading side.  That a chunk is there is told by a count in shared memory, which costs a load where asking its mbarrier takes 200
// clocks; one thread says how many have been read by everyone.
struct SgReader {
  const float* base;
  volatile int *there, *read, *stuck;
  int slots, slot, asked, total;

  __device__ __forceinline__ void await(int n) {  // the next n chunks
    asked += n;
    if (*there < asked) {
      const long long t0 = clock64();
      while (*there < asked) {
        if (*stuck) break;
        if (clock64() - t0 > tc::kWaitLimitCycles) *stuck = 1;
      }
    }
    __threadfence_block();
  }
  __device__ __forceinline__ const float* next() {
    const float* at = base + slot * kSgChunk;
    if (++slot == slots) slot = 0;
    return at;
  }
  __device__ __forceinline__ void release(int n) {
    total += n;
    if (threadIdx.x == kSgThreads - 1) *read = total;
  }
};

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}

// The loading warp: asks for chunks as slots become free and counts those that have come.  `all` chunks, `per` of them a step; in a
// cluster it takes part in the layers' barriers, which count every thread.
template <int C>
__device__ __forceinline__ void sg_load(const SmallGpt& p, float* base, uint32_t full, volatile int* there, volatile int* read,
                                        volatile int* stuck, int slots, int n_layer, int per, int all) {
  const bool lead = (threadIdx.x & 31) == 0, joined = p.cluster > 1;
  const float* src = p.w;
  int issued = 0, slot = 0, chunk = 0, in_layer = 0, come = 0, come_slot = 0, come_phase = 0;
  for (int l = 0;; ++l) {
    // as far as the products in front of the layer's barrier; all of it where there is no barrier
    const int target = joined && l < p.L ? min(all, l * SgChunks<C>::kLayer + SgChunks<C>::kQ) : all;
    bool ok = true;
    if (lead) {
      long long t0 = clock64();  // of the last thing that happened
      while (come < target) {
        bool idle = true;
        if (issued < all && issued < *read + slots) {
          const int f = chunk < n_layer ? SgChunks<C>::floats(in_layer) : kSgChunk;
          tc::mbar_expect_tx(full + 8 * slot, f * 4);
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           tc::smem_u32(base + slot * kSgChunk)),
                       "l"(src), "r"(f * 4), "r"(full + 8 * slot)
                       : "memory");
          idle = false;
          src += f;
          ++issued;
          if (++slot == slots) slot = 0;
          if (++in_layer == SgChunks<C>::kLayer) in_layer = 0;
          if (++chunk == per) {
            chunk = in_layer = 0;
            src = p.w;
          }
        }
        if (come < issued && mbar_test(full + 8 * come_slot, come_phase)) {
          idle = false;
          __threadfence_block();
          *there = ++come;
          if (++come_slot == slots) {
            come_slot = 0;
            come_phase ^= 1;
          }
        }
        if (!idle) {
          t0 = clock64();
        } else if (*stuck || clock64() - t0 > tc::kWaitLimitCycles) {
          ok = false;
          break;
        }
      }
      if (!ok) {  // nothing more is loaded; the copies in flight get a bounded chance to land
        *stuck = 1;
        for (; come < issued; ++come) {
          if (!tc::mbar_wait(full + 8 * come_slot, come_phase)) break;
          if (++come_slot == slots) {
            come_slot = 0;
            come_phase ^= 1;
          }
        }
      }
    }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!ok || !joined || l >= p.L) return;
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

template <int C, int D, int M>
__global__ void __launch_bounds__(kSgThreads + 32, 1) small_gpt_kernel(const __grid_constant__ SmallGpt p) {
  using Qkvg = Product<C, 4 * C, M>;
  using Proj = Product<C, C, M>;
  using Up = Product<C, 4 * C, M>;
  using Down = Product<2 * C, C, M>;
  using Head = Product<C, 256, M>;
  using Chunks = SgChunks<C>;
  constexpr int H = C / D, kPart = D + 4;
  constexpr int kParts = M * H >= kSgWarps ? 1 : kSgWarps / (M * H);  // warps that share a (row, head)
  constexpr int kTasks = M * H * kParts;
  extern __shared__ __align__(128) float sm[];
  const int V = p.V, L = p.L, NS = p.slots;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* ring = sm;                       // [slots][kSgChunk]
  float* u = ring + NS * kSgChunk;        // [M][C]
  float* y = u + M * C;                   // [M][C]
  float* qkvg = y + M * C;                // [M][4 C]; the feed-forward's activations in the same place
  float* act = qkvg;                      // [M][2 C]
  float* csm = qkvg + M * 4 * C;          // [M][D] cos and sin of the row's position
  float* part = csm + M * D;              // attention partials [kTasks][D + 4]
  float* mixw = part + kTasks * kPart;    // [L][2][C]
  float* cand = mixw + L * 2 * C;         // [L + 1][M][C]
  float* lg = cand + (L + 1) * M * C;     // capped logits [M][V], V a multiple of 4
  float* ex = lg + M * V;                 // the draw's scratch [M][V + 33]
  unsigned* at = reinterpret_cast<unsigned*>(p.out_tok ? ex + M * (V + 33) : lg);  // [rows, or 1][max_keys] where keys are, / 16 bytes
  __shared__ __align__(8) uint64_t full[kSgMaxSlots];
  __shared__ long long traj[M], append[M];  // append: where the token's key goes, -1 where it is out of range
  __shared__ int tok[M], pos[M], n_keys[M], fresh_key[M];  // fresh_key: which key is the step's own token's, -1 where that is not the last one
  __shared__ uint32_t bits[M];  // the random words of the step's draws
  __shared__ volatile int stuck, chunks_there, chunks_read;  // a bounded wait ran out; chunks that have come, that everyone is done with
  const bool chunk = p.T > 0;
  const int rank = chunk ? blockIdx.x % p.cluster : 0, seq0 = chunk ? blockIdx.x / p.cluster : 0;
  const int first = chunk ? rank * M : blockIdx.x * M;   // first token of the chunk, or first row
  const int live = min(M, (chunk ? p.T : p.R) - first);  // rows of this CTA that exist
  const int step0 = p.step ? *p.step : 0;
  const int cap_slots = p.kv.page_table ? p.kv.max_pages * p.kv.page_tokens : p.kv.page_tokens;
  const float scale = kLog2e / sqrtf((float)D);
  // The last token's logits only: the other CTAs of the sequence have no head.
  const bool head = !p.last_only || (p.t_base + first <= p.T_all - 1 && p.T_all - 1 < p.t_base + first + live);
  const int head_blocks = head ? (V + 255) / 256 : 0;
  const int n_layer = L * Chunks::kLayer, n_chunks = n_layer + head_blocks * Chunks::kHead;

  if (tid == 0) {
    for (int i = 0; i < NS; ++i) tc::mbar_init(tc::smem_u32(&full[i]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc::fence_async_smem();
    stuck = chunks_there = chunks_read = 0;
  }
  __syncthreads();
  const bool resident = n_chunks <= NS;  // everything fits: loaded once
  if (warp == kSgWarps) {
    sg_load<C>(p, ring, tc::smem_u32(full), &chunks_there, &chunks_read, &stuck, NS, n_layer, n_chunks, resident ? n_chunks : n_chunks * p.n_steps);
    return;
  }
  SgReader w_ring{ring, &chunks_there, &chunks_read, &stuck, NS, 0, 0, 0};

  // ---- what does not change from step to step ----
  auto key_at = [&](int seq, int slot) -> unsigned {  // a slot's place in units of 16 bytes
    const int lp = p.kv.page_table ? slot / p.kv.page_tokens : 0;
    const long long pg = p.kv.page_table ? (long long)p.kv.page_table[(long long)seq * p.kv.max_pages + lp] : (long long)seq;
    if (p.kv.page_table && (pg < 0 || (p.kv.n_pages > 0 && pg >= p.kv.n_pages))) return kNoKey;
    return (unsigned)((pg * p.kv.page_stride + (long long)(slot - lp * p.kv.page_tokens) * D) / 4);
  };
  int r_pos = 0, r_slot = 0, r_len0 = 0, r_start = 0, r_len1 = 0;
  if (tid < M && tid < live) {
    const int seq = chunk ? seq0 : first + tid, t = chunk ? p.t_base + first + tid : 0;
    tok[tid] = p.ids[chunk ? seq0 * p.T_all + t : first + tid];
    traj[tid] = p.traj ? p.traj[seq] : 0;
    r_pos = p.pos0[seq] + step0 + t;
    r_slot = p.slot0[seq] + step0 + t;
    if (p.len1) {
      r_len0 = p.len0 ? p.len0[seq] : 0;
      r_start = p.start1 ? p.start1[seq] : 0;
      r_len1 = p.len1[seq] + step0;
    } else {
      r_len1 = r_slot + 1;
    }
    r_len0 = max(0, min(r_len0, min(cap_slots, p.max_keys)));
    r_start = max(0, min(r_start, cap_slots));
  }
  // where every key that a row will ever see lies
  for (int m = 0; m < (chunk ? 1 : live); ++m) {
    const int seq = chunk ? seq0 : first + m;
    int a = 0, b = 0, n = 0;
    if (p.len1) {
      a = max(0, min(p.len0 ? p.len0[seq] : 0, min(cap_slots, p.max_keys)));
      b = max(0, min(p.start1 ? p.start1[seq] : 0, cap_slots));
      n = min(p.len1[seq] + step0 + p.n_steps - 1, cap_slots - b);
    } else {
      n = min(p.slot0[seq] + step0 + p.t_base + p.T, cap_slots);
    }
    n = min(a + max(n, 0), p.max_keys);
#pragma unroll 1
    for (int i = tid; i < n; i += kSgThreads) at[m * p.max_keys + i] = key_at(seq, i < a ? i : b + (i - a));
  }
#pragma unroll 1
  for (int i = tid; i < L * 2 * C; i += kSgThreads) mixw[i] = __ldg(p.w + p.n_w + i);
  sg_sync();
  bool lost = false;  // a wait ran out.  Every thread goes by the same answer, so that those that leave do not leave others at a barrier.
#pragma unroll 1
  for (int it = 0; it < p.n_steps; ++it) {
    if (resident) w_ring.slot = w_ring.asked = 0;
    if (tid < M) {
      const int at_slot = r_slot + it;
      const int n = r_len0 + max(0, min(r_len1 + it, cap_slots - r_start));
      const bool in = tid < live && r_pos + it >= 0 && r_pos + it < p.table_len && at_slot >= 0 && at_slot < cap_slots;
      // the newest key's place, unless the caller appends elsewhere
      const bool newest = !chunk && n <= p.max_keys && n > r_len0 && r_start + r_len1 + it - 1 == at_slot;
      const unsigned to = !in ? kNoKey : newest ? at[tid * p.max_keys + n - 1] : key_at(chunk ? seq0 : first + tid, at_slot);
      if (tid < live && (!in || n > p.max_keys)) atomicExch(p.status, 1);
      pos[tid] = in ? r_pos + it : 0;
      append[tid] = to == kNoKey ? -1 : 4ll * to;
      n_keys[tid] = tid < live ? min(n, p.max_keys) : 0;
      fresh_key[tid] = in && newest ? n - 1 : -1;
    }
    sg_sync();
    // ---- embedding and its norm; cos and sin of the positions ----
    if (warp < M) {
      const int id = warp < live ? min(max(tok[warp], 0), V - 1) : 0;
      const float cs = lane < D ? __ldg(p.cs + (long long)pos[warp] * D + lane) : 0.f;
      float x[C / 32], ss = 0.f;
#pragma unroll
      for (int i = 0; i < C / 32; ++i) {
        x[i] = __ldg(p.emb + (long long)id * C + lane + 32 * i);
        ss = fmaf(x[i], x[i], ss);
      }
      if (lane < D) csm[warp * D + lane] = cs;
      ss = warp_sum(ss);
      const float inv = rsqrtf(ss / (float)C + kRmsEps);
#pragma unroll
      for (int i = 0; i < C / 32; ++i) cand[warp * C + lane + 32 * i] = x[i] * inv;
    }
    if (p.out_tok && warp == kSgWarps - 1 && lane < live)  // where most warps have nothing to do
      bits[lane] = philox4x32_10((uint32_t)traj[lane], (uint32_t)((unsigned long long)traj[lane] >> 32), (uint32_t)(step0 + it + 1), 0u, p.seed_lo,
                                 p.seed_hi);
    __syncwarp();
    unsigned committed = 1u;
    int mult0 = 1;
#pragma unroll 1
    for (int l = 0; l < L; ++l) {
      if (warp < M) mix_row<C, M>(cand, warp, l == 0 ? 1u : committed | (1u << l), mult0, mixw + l * 2 * C, u);
      bool fresh = false;  // the running block sum starts anew
      if ((l + 1) % p.layers_per_block == 0) {
        if (l == 0) mult0 = 2;
        else committed |= 1u << l;
        fresh = true;
      }
      sg_sync();
      Qkvg::run(w_ring, u, [&](int m, int n, float v, bool mine) {
        if (mine) qkvg[m * 4 * C + n] = v;
      });
      sg_sync();
      w_ring.release(Qkvg::kGroup);
      const float* kb = static_cast<const float*>(p.kv.k) + l * p.layer_stride;
      const float* vb = static_cast<const float*>(p.kv.v) + l * p.layer_stride;
      KeyRound<D> round;
      // the first keys of this warp's first task do not depend on the token at hand (in a chunk they do, and where its key lies among them)
      if (const int w = tid_here() >> 5, m = w / kParts / H; w < kTasks && m < live && fresh_key[m] >= 0) {
        const long long o = (long long)(w / kParts % H) * p.kv.head_stride;
        round.load(at + m * p.max_keys, n_keys[m], kb + o, vb + o, qkvg, qkvg, fresh_key[m], (w % kParts) * KeyRound<D>::G * KeyRound<D>::U);
      }
      // ---- rotation, norm over the head, append ----
      constexpr int kHalf = D / 2;
#pragma unroll 1
      for (int i = tid_here(); i < M * C; i += kSgThreads) {  // a pair of q, or one of k and of v; M C is a multiple of 32
        const int m = i / C, r = i - m * C, is_k = r >= C / 2, e = r - is_k * (C / 2), h = e / kHalf, pr = e - h * kHalf;
        float* src = qkvg + m * 4 * C + is_k * C + h * D + 2 * pr;
        const float2 x = *reinterpret_cast<const float2*>(src);
        const float2 cs = *reinterpret_cast<const float2*>(csm + m * D + 2 * pr);
        const float a = x.x * cs.x - x.y * cs.y, b = x.x * cs.y + x.y * cs.x;
        float ss = a * a + b * b;
#pragma unroll
        for (int o = kHalf >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float inv = rsqrtf(ss / (float)D + kRmsEps);
        const float2 out = make_float2(a * inv, b * inv);
        if (!is_k) {
          *reinterpret_cast<float2*>(src) = make_float2(out.x * scale, out.y * scale);
        } else {
          *reinterpret_cast<float2*>(src) = out;
          if (append[m] >= 0) {
            const long long off = append[m] + (long long)h * p.kv.head_stride + 2 * pr;
            *reinterpret_cast<float2*>(const_cast<float*>(kb) + off) = out;
            *reinterpret_cast<float2*>(const_cast<float*>(vb) + off) = *reinterpret_cast<const float2*>(src + C);
          }
        }
      }
      if (chunk && p.cluster > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      } else {
        sg_sync();
      }
      // ---- attention ----
#pragma unroll 1
      for (int task = tid_here() >> 5; task < kTasks; task += kSgWarps) {
        const int pair = task / kParts, sp = task % kParts, m = pair / H, h = pair % H;
        if (m >= live) continue;
        const unsigned* keys = at + (chunk ? 0 : m * p.max_keys);
        const int n = n_keys[m], newest = fresh_key[m];  // taken from where it has just been made
        const float* row = qkvg + m * 4 * C + h * D;
        const float *kh = kb + (long long)h * p.kv.head_stride, *vh = vb + (long long)h * p.kv.head_stride;
        if (newest < 0 || task >= kSgWarps) round.load(keys, n, kh, vh, row + C, row + 2 * C, newest, sp * KeyRound<D>::G * KeyRound<D>::U);
        attend<D>(keys, n, kh, vh, round, row, row + C, row + 2 * C, newest, sp, kParts, part + task * kPart);
      }
      sg_sync();
#pragma unroll 1
      for (int i = tid_here(); i < M * C; i += kSgThreads) {
        const int m = i / C, c = i - m * C, h = c / D, d = c - h * D;
        float v = 0.f;
        if (m < live) {
          const float* src = part + (m * H + h) * kParts * kPart;
          float top = -INFINITY, sum = 0.f;
#pragma unroll
          for (int s = 0; s < kParts; ++s) top = fmaxf(top, src[s * kPart + D]);
#pragma unroll
          for (int s = 0; s < kParts; ++s) {
            const float f = top == -INFINITY ? 0.f : exp2_fast(src[s * kPart + D] - top);
            v = fmaf(f, src[s * kPart + d], v);
            sum = fmaf(f, src[s * kPart + D + 1], sum);
          }
          const float g = qkvg[m * 4 * C + 3 * C + c];
          v = (sum > 0.f ? __fdividef(v, sum) : 0.f * v) * __fdividef(1.f, 1.f + __expf(-g));  // no keys: 0; not a number stays that
        }
        y[i] = v;
      }
      sg_sync();
      float* now = cand + (l + 1) * M * C;
      const float* before = cand + l * M * C;
      Proj::run(w_ring, y, [&](int m, int n, float v, bool mine) {
        if (mine) now[m * C + n] = fresh ? v : before[m * C + n] + v;
      });
      sg_sync();
      w_ring.release(Proj::kGroup);
      if (warp < M) mix_row<C, M>(cand, warp, committed | (1u << (l + 1)), mult0, mixw + l * 2 * C + C, u);
      sg_sync();
      Up::run(w_ring, u, [&](int m, int n, float v, bool mine) {
        const float lin = fminf(fmaxf(__shfl_xor_sync(0xffffffffu, v, Up::KS), -p.limit), p.limit), g = fminf(v, p.limit);
        if (mine && (n & 1) == 0) act[m * 2 * C + (n >> 1)] = g * __fdividef(1.f, 1.f + __expf(-(p.alpha * g))) * (lin + 1.f);
      });
      sg_sync();
      w_ring.release(Up::kGroup);
      Down::run(w_ring, act, [&](int m, int n, float v, bool mine) {
        if (mine) now[m * C + n] += v;
      });
      lost = sg_any(stuck);
      w_ring.release(Down::kGroup);
      if (lost) break;
    }
    if (lost) break;
    if (!head) continue;  // (a chunk has one step)
    // ---- head: one token's logits a row ----
    if (warp < M) mix_row<C, M>(cand, warp, 1u << L, 1, nullptr, u);
    sg_sync();
#pragma unroll 1
    for (int nb = 0; nb < head_blocks; ++nb) {
      Head::run(w_ring, u, [&](int m, int n_, float v, bool mine) {
        const int n = nb * 256 + n_;
        if (!mine || n >= V || m >= live) return;
        float* out = chunk ? p.logits + (p.last_only ? (long long)seq0 : (long long)seq0 * p.T_all + p.t_base + first + m) * V
                           : p.logits + (long long)(first + m) * V;
        if (!p.last_only || p.t_base + first + m == p.T_all - 1) out[n] = p.logit_cap > 0.f ? p.logit_cap * tanhf(v / p.logit_cap) : v;
        if (p.out_tok) lg[m * V + n] = p.cap > 0.f ? softcap_value<float>(v, p.cap) : v;  // by all threads; the draw's warp takes them as they are
      });
      sg_sync();
      w_ring.release(Head::kGroup);
    }
    if (p.out_tok) {
      if (warp < live) {
        const int r = first + warp, col = step0 + it + 1;
        int t = p.force ? p.force[(long long)(r / p.force_rows) * p.force_stride + col] : -1;
        const bool plain = p.top_p >= 1.f || p.temperature == 0.f;
        if (t >= 0) {
        } else if (plain && p.log2c <= 3)
          t = draw_row<8>(lg + warp * V, V, p.temperature, bits[warp]);
        else if (plain && p.log2c == 4)
          t = draw_row<16>(lg + warp * V, V, p.temperature, bits[warp]);
        else
          t = sample_row<float>(lg + warp * V, false, ex + warp * (V + 33), V, p.log2c, 0.f, p.temperature, p.top_p, p.seed_lo, p.seed_hi,
                                traj[warp], col);
        if (lane == 0) {
          tok[warp] = t;
          p.hist[(long long)r * p.hist_stride + col] = t;
          if (it + 1 == p.n_steps) p.out_tok[r] = t;
        }
      }
      sg_sync();
    }
  }
  if (stuck && tid == 0) atomicExch(p.status, 2);
}

constexpr size_t kSgRest = 128 * 1024;  // the most that may stand next to the ring, which then has six slots

// Bytes next to the ring.
inline size_t small_gpt_smem(int C, int M, int L, int H, int V, bool draw, int keys, bool chunk) {
  const int D = C / H, tasks = M * H > kSgWarps ? M * H : kSgWarps;
  size_t f = (size_t)M * (6 * C + D) + (size_t)tasks * (D + 4) + (size_t)L * 2 * C + (size_t)(L + 1) * M * C;
  if (draw) f += (size_t)M * V + (size_t)M * (V + 33);
  f += (size_t)(chunk ? 1 : M) * keys;
  return f * sizeof(float);
}

template <int C, int D, int M>
static int small_gpt_launch(SmallGpt p, int grid, cudaStream_t st) {
  auto kern = small_gpt_kernel<C, D, M>;
  const size_t rest = small_gpt_smem(C, M, p.L, C / D, p.V, p.out_tok != nullptr, p.max_keys, p.T > 0), slot = kSgChunk * sizeof(float);
  const int n_chunks = p.L * SgChunks<C>::kLayer + (p.V + 255) / 256 * SgChunks<C>::kHead;
  p.slots = (int)((226 * 1024 - rest) / slot);  // static shared memory is under 1 KB
  if (p.slots > kSgMaxSlots) p.slots = kSgMaxSlots;
  if (p.slots > n_chunks) p.slots = n_chunks;
  const size_t smem = rest + p.slots * slot;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess && p.cluster > 8) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) {
    set_error("small_gpt: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    return DGPT_E_CUDA;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kSgThreads + 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.cluster > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, p);
  return launch_status("small_gpt");
}

template <int C>
static int small_gpt_pick(const SmallGpt& p, int M, int grid, cudaStream_t st) {
#define DGPT_SG(DD)                                                \
  do {                                                             \
    if (M == 1) return small_gpt_launch<C, DD, 1>(p, grid, st);    \
    if (M == 2) return small_gpt_launch<C, DD, 2>(p, grid, st);    \
    if (M == 4) return small_gpt_launch<C, DD, 4>(p, grid, st);    \
    return small_gpt_launch<C, DD, 8>(p, grid, st);                \
  } while (0)
  const int D = C / p.H;
  if (D == 8) DGPT_SG(8);
  if (D == 16) DGPT_SG(16);
  DGPT_SG(32);
#undef DGPT_SG
}

int small_gpt_32(const SmallGpt& p, int M, int grid, cudaStream_t st);
int small_gpt_64(const SmallGpt& p, int M, int grid, cudaStream_t st);
int small_gpt_128(const SmallGpt& p, int M, int grid, cudaStream_t st);

}  // namespace dgpt
