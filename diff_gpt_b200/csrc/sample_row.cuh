// The draw of one row by one warp: soft-cap, top-p filter and temperature sampling, the part shared by the sampling kernel and by the
// kernel that runs whole steps of a small model.
#pragma once

#include "sampling.cuh"

namespace dgpt {

struct ArgMax {
  float v;
  int i;
};
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}

// Which lane's chunk an inverse-CDF walk ends in, and how far into it: the first lane with mass whose inclusive sum lies above
// `tgt`; the last lane with mass where the rounded target reaches the total.  A lane's chunk begins at incl - mine, which is
// rounded and may lie above the previous lane's inclusive sum: a target in that gap belongs to the chunk's first token, so the
// distance is clamped at 0.  (Asked for excl <= tgt as well, such a target had no owner, about one draw in a million.)
// Returns -1 where no lane has mass or the target is not a number; `local` = INFINITY takes the chunk's last token.
__device__ __forceinline__ int walk_owner(float mine, float incl, float tgt, float* local) {
  const unsigned above = __ballot_sync(0xffffffffu, mine > 0.f && tgt < incl);
  const unsigned mass = __ballot_sync(0xffffffffu, mine > 0.f && tgt == tgt);
  *local = above ? fmaxf(tgt - (incl - mine), 0.f) : INFINITY;
  return above ? __ffs(above) - 1 : 31 - __clz(mass);
}

// Same rule and same draw as sample_kernel with shuffles only (no block barriers).  exp(z - max) of the row lives in shared memory,
// `e` [V + 33]; token i sits at word i + (i >> log2c), where 32 << log2c >= V, so that both the strided sweeps and the per-lane
// contiguous chunks (needed where token order matters) are free of bank conflicts.  The bisection stops as soon as all keys left in
// the bracket are equal, which takes about log2(distinct keys) sweeps instead of 30.
// `vec_ok`: the row is 16-byte aligned and V a multiple of 16 bytes.  `step` keys the random stream with `traj`.
template <typename T>
__device__ __forceinline__ int sample_row(const T* row, bool vec_ok, float* e, int V, int log2c, float cap, float temperature, float top_p,
                                          uint32_t seed_lo, uint32_t seed_hi, long long traj, int step) {
  const int lane = threadIdx.x & 31;
  auto at = [&](int i) -> float& { return e[i + (i >> log2c)]; };
  ArgMax best{-INFINITY, 0x7fffffff};
  constexpr int VEC = Io<T>::kVec16;
  if (vec_ok) {
    // 16-byte loads, four in flight per lane; a lane visits its tokens in increasing order, so `>`
    // keeps the lowest index among equal values, and `better` does the same across lanes
    const int n_vec = V / VEC;
    for (int j0 = lane; j0 < n_vec; j0 += 128) {
      float x[4][VEC];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j0 + 32 * u < n_vec) ld16<T>(row + (j0 + 32 * u) * VEC, x[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (j0 + 32 * u >= n_vec) continue;
        const int i0 = (j0 + 32 * u) * VEC;
#pragma unroll
        for (int k = 0; k < VEC; ++k) {
          float v = x[u][k];
          if (cap > 0.f) v = softcap_value<T>(v, cap);
          at(i0 + k) = v;
          if (v > best.v) best = ArgMax{v, i0 + k};
        }
      }
    }
  } else {
    for (int i = lane; i < V; i += 32) {
      float x = Io<T>::ld(row + i);
      if (cap > 0.f) x = softcap_value<T>(x, cap);
      at(i) = x;
      if (x > best.v) best = ArgMax{x, i};
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax t;
    t.v = __shfl_xor_sync(0xffffffffu, best.v, o);
    t.i = __shfl_xor_sync(0xffffffffu, best.i, o);
    best = better(best, t);
  }
  int token = best.i;
  if (temperature != 0.f) {
    const float zmax = best.v;
    float p4[4] = {0.f, 0.f, 0.f, 0.f};  // four running sums: consecutive adds do not wait on one another
    int i = lane;
    for (; i + 96 < V; i += 128) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float ev = __expf(at(i + 32 * u) - zmax);
        at(i + 32 * u) = ev;
        p4[u] += ev;
      }
    }
    for (; i < V; i += 32) {
      const float ev = __expf(at(i) - zmax);
      at(i) = ev;
      p4[0] += ev;
    }
    const float Z = warp_sum((p4[0] + p4[1]) + (p4[2] + p4[3]));
    const bool filt = top_p < 1.f;
    uint32_t key_b = 0u;
    int i_cut = V;
    const int chunk = 1 << log2c;
    const int c0 = lane * chunk, c1 = min(V, c0 + chunk);  // this lane's tokens where order matters
    // Fast path (rejection sampling): draw from softmax(z / T) over ALL tokens and accept the token if
    // it lies in the nucleus, i.e. if the mass ranked before it is below top_p.  Accepted draws follow
    // exactly the restricted distribution, and a draw costs two sweeps instead of a full boundary
    // search.  Attempt a uses Philox counter word 3 = a.  If kAttempts draws are rejected (a high
    // temperature over a tiny nucleus), the exact boundary is computed below.
    constexpr int kAttempts = 8;
    bool done = false;
    {
      __syncwarp();  // chunks below were written by other lanes
      const float inv_t = 1.f / temperature;
      const bool t1 = temperature == 1.f;
      float mine = 0.f;
      for (int i = c0; i < c1; ++i) {
        const float ev = at(i);
        mine += t1 ? ev : __expf(__logf(ev) * inv_t);
      }
      float incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      const float W = __shfl_sync(0xffffffffu, incl, 31);
      const float target = fmaxf(top_p, 1e-30f) * Z;
      for (int a = 0; a < kAttempts && !done; ++a) {
        const uint32_t bits = philox4x32_10((uint32_t)traj, (uint32_t)((unsigned long long)traj >> 32),
                                            (uint32_t)step, (uint32_t)a, seed_lo, seed_hi);
        const float tgt = (float)(bits >> 8) * (1.0f / 16777216.0f) * W;
        float local;
        const int who = walk_owner(mine, incl, tgt, &local);
        int pick = best.i;
        if (lane == who) {
          float c = 0.f;
          for (int i = c0; i < c1; ++i) {
            const float ev = at(i);
            const float w = t1 ? ev : __expf(__logf(ev) * inv_t);
            c += w;
            if (w > 0.f) pick = i;
            if (w > 0.f && c > local) break;
          }
        }
        pick = __shfl_sync(0xffffffffu, pick, max(who, 0));
        if (!filt) {
          token = pick;
          done = true;
          break;
        }
        const float ek = at(pick);
        const uint32_t kk = __float_as_uint(ek);
        float a4[4] = {0.f, 0.f, 0.f, 0.f}, before = 0.f;
        int i = lane;
        for (; i + 96 < V; i += 128) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float ev = at(i + 32 * u);
            const uint32_t k = __float_as_uint(ev);
            a4[u] += k > kk ? ev : 0.f;
            before += (k == kk && i + 32 * u < pick) ? 1.f : 0.f;
          }
        }
        for (; i < V; i += 32) {
          const float ev = at(i);
          const uint32_t k = __float_as_uint(ev);
          a4[0] += k > kk ? ev : 0.f;
          before += (k == kk && i < pick) ? 1.f : 0.f;
        }
        float above = warp_sum((a4[0] + a4[1]) + (a4[2] + a4[3]));
        before = warp_sum(before);
        if (above + before * ek < target) {
          token = pick;
          done = true;
        }
      }
    }
    if (done) {
      // nothing left to do
    } else if (filt) {
      const float target = fmaxf(top_p, 1e-30f) * Z;
      uint32_t lo = 0u, hi = 0x3f800000u;  // mass above lo >= target, mass above hi = 0 < target
      while (hi - lo > 1u) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        float s = 0.f;
        uint32_t kmn = 0xffffffffu, kmx = 0u;
        for (int i = lane; i < V; i += 32) {
          const float ev = at(i);
          const uint32_t k = __float_as_uint(ev);
          if (k > lo && k <= hi) {
            kmn = min(kmn, k);
            kmx = max(kmx, k);
          }
          s += k > mid ? ev : 0.f;
        }
        s = warp_sum(s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          kmn = min(kmn, __shfl_xor_sync(0xffffffffu, kmn, o));
          kmx = max(kmx, __shfl_xor_sync(0xffffffffu, kmx, o));
        }
        if (kmn == kmx) {  // a single key value is left in (lo, hi]: it is the boundary
          hi = kmn;
          break;
        }
        if (s < target) hi = mid; else lo = mid;
      }
      uint32_t kmin = 0xffffffffu;
      for (int i = lane; i < V; i += 32) {
        const uint32_t k = __float_as_uint(at(i));
        if (k >= hi) kmin = min(kmin, k);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) kmin = min(kmin, __shfl_xor_sync(0xffffffffu, kmin, o));
      key_b = kmin;
      float above = 0.f, cnt = 0.f;
      for (int i = lane; i < V; i += 32) {
        const float ev = at(i);
        const uint32_t k = __float_as_uint(ev);
        above += k > key_b ? ev : 0.f;
        cnt += k == key_b ? 1.f : 0.f;
      }
      above = warp_sum(above);
      cnt = warp_sum(cnt);
      int keep = (int)ceilf((target - above) / __uint_as_float(key_b));
      keep = max(1, min(keep, (int)cnt));
      if (keep < (int)cnt) {  // id of the keep-th token (in id order) whose key equals key_b
        __syncwarp();  // chunks below were written by other lanes
        int mine = 0;
        for (int i = c0; i < c1; ++i) mine += __float_as_uint(at(i)) == key_b ? 1 : 0;
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        const int excl = incl - mine;
        int found = V - 1;
        const bool own = excl < keep && keep <= incl;
        if (own) {
          int seen = excl;
          for (int i = c0; i < c1; ++i)
            if (__float_as_uint(at(i)) == key_b && ++seen == keep) {
              found = i;
              break;
            }
        }
        const unsigned who = __ballot_sync(0xffffffffu, own);
        i_cut = __shfl_sync(0xffffffffu, found, who ? __ffs(who) - 1 : 0);
      }
    }
    // exact path: inverse-CDF draw in token order over the kept tokens
    if (!done) {
    __syncwarp();  // chunks below were written by other lanes
    const float inv_t = 1.f / temperature;
    float mine = 0.f;
    for (int i = c0; i < c1; ++i) {
      const float ev = at(i);
      bool kept = true;
      if (filt) {
        const uint32_t k = __float_as_uint(ev);
        kept = k > key_b || (k == key_b && i <= i_cut);
      }
      const float w = !kept ? 0.f : (temperature == 1.f ? ev : __expf(__logf(ev) * inv_t));
      at(i) = w;
      mine += w;
    }
    float incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const float W = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t bits = philox4x32_10((uint32_t)traj, (uint32_t)((unsigned long long)traj >> 32),
                                        (uint32_t)step, (uint32_t)kAttempts, seed_lo, seed_hi);
    const float u = (float)(bits >> 8) * (1.0f / 16777216.0f);
    const float tgt = u * W;
    float local;
    const int who = walk_owner(mine, incl, tgt, &local);
    int pick = best.i;
    if (lane == who) {
      float c = 0.f;
      for (int i = c0; i < c1; ++i) {
        const float w = at(i);
        c += w;
        if (w > 0.f) pick = i;
        if (w > 0.f && c > local) break;
      }
    }
    token = __shfl_sync(0xffffffffu, pick, max(who, 0));
    }
  }
  return token;
}

}  // namespace dgpt
