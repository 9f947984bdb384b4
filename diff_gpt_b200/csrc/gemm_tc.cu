// tcgen05 / TMEM GEMM for the linear layers of the decode step (sm_100a), with the SwiGLU of the
// feed-forward block in its epilogue.
//
//   acc[m, n] = sum_k A[m, k] * W[n, k]        A: activations [M, K] bf16, W: nn.Linear weight [N, K] bf16
//   mode 0:  out[m, n]     = bf16(acc[m, n])
//   mode 1:  out[m, n / 2] = swiglu(bf16(acc[m, n]), bf16(acc[m, n + 1]))   for even n  (interleaved gate / linear)
//   mode 2:  out[m, n]     = bf16(resid[m, n] + acc[m, n])                    (the residual add of addmm, one rounding)
//   mode 4:  out[m, n]     = bf16(xielu(acc[m, n]))   with alpha_p = alpha, alpha_n = limit
//   mode 5:  out[m, n / 2] = bf16(silu(acc[m, n]) * acc[m, n + 1])   for even n  (interleaved gate / up)
//   mode 6:  out[m, n]     = cap(bf16(acc[m, n]))   with cap = alpha: the head of a scoring forward, its soft-cap applied on the
//            way out (a pass of its own over the stored logits took 214 us for 131072 x 512 of them)
//   mode 3:  nothing is stored: row m keeps the best key of  key[m, n] = cap(bf16(acc[m, n])) / T + Gumbel noise(m, n)
//            (no noise and T = 1 for an arg-max) in best[m], a 64-bit word (order-preserving key bits, ~n) raised with
//            atomicMax - the tied-embedding head with the draw in its epilogue, so [M, N] logits never reach HBM
//
// Persistent, warp-specialised CTAs of 576 threads, one per SM.  A tile is 128 CG x BN outputs, made by one CTA (CG = 1, BN = 64 to 256)
// or by a CTA pair (CG = 2, BN = 128 to 256: one tcgen05.mma of M = 256 over both SMs; each CTA stages its 128 rows of A and half of the W
// rows, so a pair reads W once where two single CTAs read it twice).  Tiles are taken round robin, eight rows of tiles at a time, so that
// what is in flight shares both operands in L2:
//   warp 17, lane 0 loader: TMA loads of the A and W blocks (64 of K), 128-byte swizzle, a ring of up to 8 stages; both CTAs of a
//                   pair report their bytes to the leader's barrier
//   warp 16, lane 0 issuer (of the leader): four tcgen05.mma (K 16) per block into one of two TMEM accumulators
//   warps 0-15      epilogue: a unit is the 32 rows (TMEM lanes) that a warp can reach by 64 columns; a warp reads its unit 32 columns at a time, applies the
//                   epilogue, packs bf16 into its swizzled staging tile and has TMA store it
// so the epilogue of tile i runs while the tensor cores work on tile i + 1.  No multicast load.
// What bounds it: the tensor cores under the power limit where K is long, and the epilogue's instructions where K is a few
// blocks (128 x 64 multiply-adds per output at K = 256 leave about 30 clocks of one scheduler for it).  Hence 16 warps rather than
// 8, one-instruction exponentials and reciprocals, and packed conversions (a lone cvt to bf16 runs at a quarter of the rate; the
// SwiGLU has five).  Measured in us, single CTAs of 8 epilogue warps that stored from their lanes -> this: 8192 x 16384 x 2048 plain
// 489 -> 367 (1500 TFLOP/s), 16384 x 5472 x 1024 SiLU gate 195 -> 135, 65536 x 8192 x 2048 xIELU 1685 -> 1565, 131072 x 10912 x 2048
// SiLU gate 4981 -> 4000, 228480 x 2048 x 512 SwiGLU 609 -> 421, 131072 x 1024 x 256 SwiGLU 154 -> 88, 4096 x 3072 x 768 SwiGLU
// 25.0 -> 20.9; 8 warps with the pairs: 561, 169 and 27.0 for the last three.
// Every mbarrier wait is bounded; a wait that runs out raises a CTA-wide abort flag, is reported through
// the status word, and every role drains what it issued before TMEM is freed.
#include "activation.cuh"
#include "linear.cuh"
#include "sampling.cuh"
#include "tcgen05.cuh"

namespace dgpt {
namespace tc {

constexpr int kGM = 128, kGK = 64;  // rows per CTA, K per stage
constexpr uint32_t kGABytes = kGM * 128;
constexpr int kGEpiWarps = 16;
constexpr int kGThreads = 32 * (kGEpiWarps + 2);  // and the MMA issuer's warp, the loader's warp
constexpr int kGGroupM = 8;             // rows of tiles that are walked together
constexpr uint32_t kGSmemMax = 232448;  // shared memory one CTA can have
constexpr uint32_t kGSmemFixed = 1024 + 512;  // alignment of the ring, barriers
__host__ __device__ constexpr uint32_t gemm_idesc(int m, int bn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__host__ __device__ constexpr bool epi_halves(int epi) { return epi == 1 || epi == 5; }  // column pairs become one output
__host__ __device__ constexpr uint32_t epi_tile_bytes(int epi) { return epi == 3 ? 0u : epi_halves(epi) ? 32u * 64u : 32u * 128u; }
__host__ __device__ constexpr uint32_t gemm_stage_bytes(int bn, int cg) { return kGABytes + (uint32_t)(bn / cg) * 128u; }
__host__ __device__ constexpr int gemm_stages(int bn, int cg, int epi) {
  const uint32_t n = (kGSmemMax - kGSmemFixed - kGEpiWarps * epi_tile_bytes(epi)) / gemm_stage_bytes(bn, cg);
  return n > 8 ? 8 : (int)n;
}
__host__ __device__ constexpr uint32_t gemm_smem(int bn, int cg, int epi) {
  return kGSmemFixed + kGEpiWarps * epi_tile_bytes(epi) + (uint32_t)gemm_stages(bn, cg, epi) * gemm_stage_bytes(bn, cg);
}

struct GemmParams {
  const __nv_bfloat16* resid;  // epilogue 2: added to the accumulator before the one rounding (may alias out)
  long long resid_rs;
  int M, N, K;
  float alpha, limit;
  int* status;
  HeadDraw draw;  // epilogue 3
};

// order-preserving map of a float onto unsigned integers
__device__ __forceinline__ uint32_t float_order_bits(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// `bar` is an address of the cluster: this CTA's own barrier, or (CG = 2) that of the pair's leader
template <int CG>
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  if constexpr (CG == 2)
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(c0), "r"(c1)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// One block of 64 along K: four MMAs whose descriptors advance by 32 bytes; the first takes the accumulate flag.
template <int CG>
__device__ __forceinline__ void gemm_mma_block(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  if constexpr (CG == 2)
    asm volatile(
        "{\n\t.reg .pred p0, pt;\n\t.reg .b64 a, b;\n\t"
        "setp.ne.b32 p0, %4, 0;\n\tsetp.eq.b32 pt, 0, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p0;\n\t"
        "add.u64 a, %1, 2;\n\tadd.u64 b, %2, 2;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, pt;\n\t"
        "add.u64 a, %1, 4;\n\tadd.u64 b, %2, 4;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, pt;\n\t"
        "add.u64 a, %1, 6;\n\tadd.u64 b, %2, 6;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, pt;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
  else
    umma_ss4<2, 2>(d, a, b, idesc, acc);
}
// Arrives at the barrier (of both CTAs of a pair) once all MMAs issued so far have finished.
template <int CG>
__device__ __forceinline__ void gemm_commit(uint32_t bar) {
  if constexpr (CG == 2)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3)
                 : "memory");
  else
    umma_commit(bar);
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t in_leader(uint32_t addr) {  // the same shared-memory address in the cluster's first CTA
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ uint32_t in_other(uint32_t addr, uint32_t rank) {  // and in the pair's other CTA
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank ^ 1u));
  return r;
}
__device__ __forceinline__ void store_cluster(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
template <int CG>
__device__ __forceinline__ void sync_ctas() {
  if constexpr (CG == 2) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
}

struct GemmTile {
  int m, n;
};
// Tile `t` in the order of the walk: kGGroupM rows of tiles at a time, down the rows before the next column.
__device__ __forceinline__ GemmTile gemm_tile(int t, int tiles_m, int tiles_n) {
  const int per = kGGroupM * tiles_n, g = t / per, first = g * kGGroupM;
  const int rows = min(kGGroupM, tiles_m - first), i = t - g * per;
  const int n = i / rows;
  return {first + i - n * rows, n};
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// EPI is a compile-time choice, so that no epilogue carries another's registers and branches (with the mode tested at run time
// the feed-forward GEMM took 21.1 instead of 17.7 us on 2048 rows).
template <int BN, int CG, int EPI>
__global__ void __launch_bounds__(kGThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mw, const __grid_constant__ CUtensorMap mo,
               const GemmParams p) {
  constexpr bool kHalf = epi_halves(EPI), kDraw = EPI == 3;
  constexpr int kStages = gemm_stages(BN, CG, EPI);
  constexpr uint32_t kStageBytes = gemm_stage_bytes(BN, CG);
  constexpr uint32_t kIdesc = gemm_idesc(kGM * CG, BN);
  constexpr uint32_t kTileBytes = epi_tile_bytes(EPI);
  constexpr int kAccStride = 256;  // TMEM columns between the two accumulators
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + kStages * kStageBytes;  // a tile of 32 rows per epilogue warp
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + kGEpiWarps * kTileBytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 24);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile uint32_t* loaded = tmem_slot + 2;  // in the leader: blocks that each CTA of the pair has asked for, once it has stopped
  const uint32_t a0 = smem_u32(smem);
  const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * kStages, bar_accf = bar_empty + 8 * kStages,
                 bar_acce = bar_accf + 16, bar_drain = bar_acce + 16;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = CG == 2 ? cluster_rank() : 0u;
  const int worker = blockIdx.x / CG, workers = gridDim.x / CG;
  const int tiles_n = (p.N + BN - 1) / BN, tiles_m = (p.M + CG * kGM - 1) / (CG * kGM);
  const int n_tiles = tiles_m * tiles_n;
  const int n_kb = (p.K + kGK - 1) / kGK;

  if (tid == 0) {
    *abort_flag = 0;
    loaded[0] = loaded[1] = 0;
    for (int i = 0; i < kStages; ++i) {
      mbar_init(bar_full + 8 * i, 1);
      mbar_init(bar_empty + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_accf + 8 * i, 1);
      mbar_init(bar_acce + 8 * i, CG * 4 * (BN / 64));  // the warps that read a tile
    }
    mbar_init(bar_drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  if (warp == 0) {
    if constexpr (CG == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      tmem_alloc(smem_u32(tmem_slot), 512);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  sync_ctas<CG>();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  dep_wait();  // everything above touched only this CTA's own shared memory and TMEM

  if (warp == kGEpiWarps + 1) {
    // ================= loader =================
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&ma)) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mw)) : "memory");
      const uint32_t full = CG == 2 ? in_leader(bar_full) : bar_full;
      int last[kStages];  // parity of the newest load per slot (for the drain on failure)
      for (int i = 0; i < kStages; ++i) last[i] = -1;
      int s = 0;
      uint32_t ph = 0, blocks = 0;
      bool ok = true;
      for (int tile = worker; ok && tile < n_tiles; tile += workers) {
        const GemmTile t = gemm_tile(tile, tiles_m, tiles_n);
        const int row = (t.m * CG + (int)rank) * kGM, col = t.n * BN + (int)rank * (BN / CG);
        for (int kb = 0; kb < n_kb; ++kb) {
          ok = wait_or_abort(bar_empty + 8 * s, ph ^ 1u, abort_flag, 32);  // a fresh barrier passes parity 1
          if (!ok) break;
          const uint32_t dst = a0 + s * kStageBytes;
          // rows or columns outside the matrices are zero-filled and counted; the leader expects both CTAs' bytes
          if (rank == 0) mbar_expect_tx(bar_full + 8 * s, CG * kStageBytes);
          tma_load_2d<CG>(dst, &ma, full + 8 * s, kb * kGK, row);
          tma_load_2d<CG>(dst + kGABytes, &mw, full + 8 * s, kb * kGK, col);
          last[s] = (int)ph;
          ++blocks;
          if (++s == kStages) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      // The commits of the last MMAs arrive on bar_empty, in a pair from the other SM: the CTA stays until they have.
      for (int i = 0; ok && i < kStages; ++i)
        if (last[i] >= 0) ok = wait_or_abort(bar_empty + 8 * i, (uint32_t)last[i], abort_flag, 36);
      if (!ok || *abort_flag) {
        if (p.status) atomicExch(p.status, *abort_flag ? *abort_flag : 32);
        if (CG == 1)
          for (int i = 0; i < kStages; ++i)
            if (last[i] >= 0) mbar_wait(bar_full + 8 * i, (uint32_t)last[i]);  // bounded: let copies in flight land
      }
      if constexpr (CG == 2) store_cluster(in_leader(smem_u32(tmem_slot + 2) + 4 * rank), blocks);
    }
  } else if (warp == kGEpiWarps) {
    // ================= MMA issuer =================
    if (lane == 0 && rank == 0) {
      unsigned t_local = 0;
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = worker; ok && tile < n_tiles; tile += workers, ++t_local) {
        const int a = t_local & 1;
        ok = wait_or_abort(bar_acce + 8 * a, ((t_local >> 1) & 1u) ^ 1u, abort_flag, 33);  // epilogue has emptied it
        if (!ok) break;
        tc_fence_after();
        for (int kb = 0; kb < n_kb; ++kb) {
          ok = wait_or_abort(bar_full + 8 * s, ph, abort_flag, 34);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = a0 + s * kStageBytes;
          gemm_mma_block<CG>(tmem + a * kAccStride, smem_desc(sa, 16, 1024), smem_desc(sa + kGABytes, 16, 1024), kIdesc, kb > 0 ? 1u : 0u);
          gemm_commit<CG>(bar_empty + 8 * s);  // the slot is free once these MMAs have read it
          if (++s == kStages) {
            s = 0;
            ph ^= 1u;
          }
        }
        if (ok) gemm_commit<CG>(bar_accf + 8 * a);
      }
      if (!ok || *abort_flag) {
        if (p.status) atomicExch(p.status, *abort_flag ? *abort_flag : 34);
        gemm_commit<CG>(bar_drain);  // completes when everything issued so far has finished
        mbar_wait(bar_drain, 0);
      }
    }
  } else {
    // ================= epilogue =================
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);  // a warp reaches the TMEM lanes of its quarter only
    const uint32_t acce = CG == 2 ? in_leader(bar_acce) : bar_acce;
    const uint32_t buf = smem_u32(staging) + warp * kTileBytes;
    constexpr int kUnits = BN / 64;  // of a tile
    if (!kDraw && lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mo)) : "memory");
    unsigned t_local = 0;
    bool ok = true;
    for (int tile = worker; ok && tile < n_tiles; tile += workers, ++t_local) {
      // Unit of this warp's group: its own number, or with two units a tile groups 0 and 1 on the first accumulator's tiles, 2
      // and 3 on the second's.  Either way a group sees every phase of the barriers it waits on.
      const int u = kUnits == 2 ? (warp >> 2) - 2 * (int)(t_local & 1) : warp >> 2;
      if (u < 0 || u >= kUnits) continue;
      const GemmTile t = gemm_tile(tile, tiles_m, tiles_n);
      const int a = t_local & 1;
      ok = wait_or_abort(bar_accf + 8 * a, (t_local >> 1) & 1u, abort_flag, 35);
      ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld is warp-collective: the warp leaves together
      if (!ok) break;
      tc_fence_after();
      const int row0 = (t.m * CG + (int)rank) * kGM + (warp & 3) * 32, row = row0 + lane;
      const int col = t.n * BN + u * 64;
      const bool any = row0 < p.M && col < p.N;  // uniform in the warp
      float best_v = -INFINITY;  // epilogue 3: this thread's best key over its columns of the tile, and where
      int best_n = 0x7fffffff;
      long long traj = 0;
      int step = 0;
      if (kDraw && row < p.M) {
        traj = p.draw.traj_ids ? p.draw.traj_ids[row] : p.draw.traj_id0 + row;
        step = p.draw.step_base + (p.draw.step_ptr ? *p.draw.step_ptr : 0);
      }
      if (!kDraw) {
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the last unit's tile has been read out
        __syncwarp();
      }
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        float v[32];
        __syncwarp();
        tmem_ld32(lane_addr + a * kAccStride + u * 64 + part * 32, v);
        if (part == 1) {  // the accumulator goes back to the issuer as soon as its last columns are in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if constexpr (CG == 2) arrive_cluster(acce + 8 * a);
            else mbar_arrive(acce + 8 * a);
          }
        }
        const int c0 = col + part * 32;
        if constexpr (kDraw) {
          using B = Io<__nv_bfloat16>;
          if (!any) continue;
#pragma unroll
          for (int q = 0; q < 8; ++q) {  // four columns per random-number block
            const int n0 = c0 + 4 * q;
            if (n0 >= p.N || row >= p.M) break;  // N is a multiple of 16
            uint32_t rnd[4] = {0u, 0u, 0u, 0u};
            if (p.draw.inv_temperature > 0.f)
              philox4x32_10_words((uint32_t)traj, (uint32_t)((unsigned long long)traj >> 32), (uint32_t)step,
                                  0x80000000u | (uint32_t)(n0 >> 2), p.draw.seed_lo, p.draw.seed_hi, rnd);
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              float z = B::round(v[4 * q + x]);  // the logit as a bf16 Linear would have written it
              if (p.draw.cap > 0.f) z = softcap_value<__nv_bfloat16>(z, p.draw.cap);
              float key = z;
              if (p.draw.inv_temperature > 0.f) {
                const float u01 = ((float)(rnd[x] >> 8) + 0.5f) * (1.f / 16777216.f);  // in (0, 1)
                key = z * p.draw.inv_temperature - __logf(-__logf(u01));               // arg-max of these keys ~ softmax(z / T)
              }
              if (key > best_v) {  // columns are visited in increasing order: the lowest index wins ties
                best_v = key;
                best_n = n0 + x;
              }
            }
          }
        } else {
          if (!any) continue;
          if constexpr (EPI == 2) {
            if (row < p.M) {
              const __nv_bfloat16* src = p.resid + (long long)row * p.resid_rs + c0;
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                if (c0 + 8 * q >= p.N) break;  // N is a multiple of 16
                float r8[8];
                ld16<__nv_bfloat16>(src + 8 * q, r8);
#pragma unroll
                for (int x = 0; x < 8; ++x) v[8 * q + x] += r8[x];
              }
            }
          }
          constexpr int kWords = kHalf ? 8 : 16;  // packed pairs of outputs
          uint32_t w[kWords];
          if constexpr (!kHalf) {
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              float lo = v[2 * k], hi = v[2 * k + 1];
              if constexpr (EPI == 4) {
                lo = xielu_fast(lo, p.alpha, p.limit);
                hi = xielu_fast(hi, p.alpha, p.limit);
              } else if constexpr (EPI == 6) {
                lo = softcap_logit(Io<__nv_bfloat16>::round(lo), p.alpha);
                hi = softcap_logit(Io<__nv_bfloat16>::round(hi), p.alpha);
              }
              w[k] = pack_bf16(lo, hi);
            }
          } else {
            using B = Io<__nv_bfloat16>;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              float r[2];
#pragma unroll
              for (int x = 0; x < 2; ++x) {
                const float gate = v[4 * k + 2 * x], up = v[4 * k + 2 * x + 1];
                if constexpr (EPI == 5) {
                  r[x] = silu_mul_fast(gate, up);
                } else {
                  // the reference's Linear writes bf16 before the activation reads it
                  const float g = fminf(B::round(gate), p.limit);
                  const float lin = fminf(fmaxf(B::round(up), -p.limit), p.limit);
                  const float sg = B::round(rcp_fast(1.f + exp_fast(-B::round(p.alpha * g))));
                  r[x] = B::round(g * sg) * B::round(lin + 1.f);
                }
              }
              w[k] = pack_bf16(r[0], r[1]);
            }
          }
          // Staging tile: 32 rows of 64 (32) outputs; the 16-byte chunk index is mixed with the row as TMA's 128-byte
          // (64-byte) swizzle wants it, which also keeps eight rows' stores of one chunk off each other's banks.
          constexpr uint32_t kPitch = kHalf ? 64u : 128u;
          const uint32_t mix = kHalf ? (lane >> 1) & 3u : lane & 7u;
#pragma unroll
          for (int q = 0; q < kWords / 4; ++q)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(buf + lane * kPitch + (((uint32_t)(part * (kWords / 4) + q) ^ mix) << 4)),
                         "r"(w[4 * q]), "r"(w[4 * q + 1]), "r"(w[4 * q + 2]), "r"(w[4 * q + 3])
                         : "memory");
        }
      }
      if (!kDraw && any) {
        fence_async_smem();
        __syncwarp();
        if (lane == 0) tma_store_2d(&mo, buf, kHalf ? col >> 1 : col, row0);  // clipped at the matrix's edges
      }
      if (kDraw && any && row < p.M && best_n != 0x7fffffff)
        atomicMax(p.draw.best + row, ((unsigned long long)float_order_bits(best_v) << 32) | (uint32_t)(~(uint32_t)best_n));
    }
    // the staging tiles are this CTA's own memory: it stays until they have been read out
    if (!kDraw && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    if (!ok && p.status && lane == 0) atomicExch(p.status, *abort_flag ? *abort_flag : 35);
  }
  tc_fence_before();
  __syncwarp();
  if (CG == 2 && lane == 0 && *abort_flag) store_cluster(in_other(smem_u32(tmem_slot + 1), rank), (uint32_t)*abort_flag);
  __syncwarp();
  sync_ctas<CG>();  // no CTA of a pair leaves while the other may still signal it or read its operands
  if (CG == 2 && *abort_flag) {  // the same in both CTAs: a wait has run out somewhere, and nobody issues copies any more
    if (rank == 0 && tid == 0) {
      // Both CTAs' copies report to the leader's barriers.  A slot's last block may have been asked for by the other CTA alone, one ahead
      // at most (the next needs that one's MMAs): its phase is still to be opened.
      for (uint32_t i = 0; i < (uint32_t)kStages; ++i) {
        const uint32_t own = (loaded[0] + kStages - 1 - i) / kStages, other = (loaded[1] + kStages - 1 - i) / kStages;
        if (other > own) mbar_expect_tx(bar_full + 8 * i, kStageBytes);
        const uint32_t n = other > own ? other : own;
        if (n > 0) mbar_wait(bar_full + 8 * i, (n - 1) & 1u);  // bounded
      }
    }
    __syncwarp();
    sync_ctas<CG>();
  }
  if (warp == 0) {
    if constexpr (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    else tmem_dealloc(tmem, 512);
  }
}

// The bounded wait by itself: two threads (of two warps) wait on a barrier that only one arrival could complete.  With
// `arrive` set the first thread arrives and both waits succeed; without it nothing ever arrives, the first
// wait gives up after `limit_cycles`, raises the flag, the second thread sees the flag and gives up too.
// out[0], out[1]: 1 where the wait succeeded; out[2]: the flag (the code of the wait that gave up);
// out[3]: clock cycles the first thread spent.
__global__ void bounded_wait_probe_kernel(int arrive, long long limit_cycles, int* out) {
  __shared__ uint64_t bar;
  __shared__ int flag;
  const uint32_t b = smem_u32(&bar);
  if (threadIdx.x == 0) {
    flag = 0;
    mbar_init(b, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0 && arrive) mbar_arrive(b);
  if (threadIdx.x == 0 || threadIdx.x == 32) {  // two warps; the second has a limit it will not reach
    const int who = threadIdx.x >> 5;
    const long long t0 = clock64();
    const bool ok = wait_or_abort(b, 0, &flag, 40 + who, who == 0 ? limit_cycles : 16 * limit_cycles);
    out[who] = ok ? 1 : 0;
    if (who == 0) out[3] = (int)min(clock64() - t0, (long long)0x7fffffff);
  }
  __syncthreads();
  if (threadIdx.x == 0) out[2] = flag;
}

// 2-D bf16 tensor map over a row-major [rows, cols] matrix with a [box_rows][box_cols] box, box_cols 64 (128-byte swizzle) or
// 32 (64-byte swizzle).
static bool encode_2d(CUtensorMap* map, const void* base, long long rows, long long cols, long long row_stride,
                      int box_rows, int box_cols = 64) {
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  if (rows == 1) row_stride = (cols + 7) / 8 * 8;  // a lone row's stride says nothing
  const cuuint64_t strides[1] = {(cuuint64_t)row_stride * 2};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  const cuuint32_t ones[2] = {1, 1};
  CUresult r = encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, ones,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("linear: cuTensorMapEncodeTiled failed with %d", (int)r);
    return false;
  }
  return true;
}

struct GemmOperands {
  const void *a, *w;
  void* out;
  long long a_rs, w_rs, out_rs;
};

template <int BN, int CG, int EPI>
static int gemm_launch(const GemmOperands& o, const GemmParams& p, int n_sm, int dev, cudaStream_t st) {
  constexpr uint32_t kSmem = gemm_smem(BN, CG, EPI);
  static_assert(kSmem <= kGSmemMax && gemm_stages(BN, CG, EPI) >= 3 && 2 * gemm_stages(BN, CG, EPI) + 5 <= 24, "shared memory of the GEMM");
  auto kernel = gemm_tc_kernel<BN, CG, EPI>;
  static bool ready[64] = {};
  if (!ready[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) {
      set_error("linear: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      return DGPT_E_CUDA;
    }
    ready[dev] = true;
  }
  CUtensorMap ma, mw, mo = {};
  const int cols = epi_halves(EPI) ? p.N / 2 : p.N;
  if (!encode_2d(&ma, o.a, p.M, p.K, o.a_rs, kGM) || !encode_2d(&mw, o.w, p.N, p.K, o.w_rs, BN / CG) ||
      (EPI != 3 && !encode_2d(&mo, o.out, p.M, cols, o.out_rs, 32, epi_halves(EPI) ? 32 : 64)))
    return DGPT_E_CUDA;
  const int tiles = ((p.M + CG * kGM - 1) / (CG * kGM)) * ((p.N + BN - 1) / BN), slots = n_sm / CG;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(CG * (tiles < slots ? tiles : slots)));
  cfg.blockDim = dim3(kGThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = dep_launch_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CG;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CG == 2 ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kernel, ma, mw, mo, p);  // errors surface through launch_status()
  return launch_status("linear");
}

// Which tile: the form with the least estimated time in clocks, rounds of tiles x clocks of one.  A k-block of 64 takes 2 BN clocks
// of the tensor cores in either form; bringing it in takes its bytes per SM at 56 a clock; an epilogue that runs beside the next tile's product
// takes about 16 clocks a column; and a pair costs 4000 more (its launch, and barriers across SMs at both ends), which single CTAs of up
// to 256 columns save where there is little to do.  Over 289 layers of 3 to 65536 rows, N 256 to 16384 and K 128 to 2048, every form measured, the
// one chosen is 0.3 % behind the best on average.  (Without the single CTAs of 256 and 192 columns, no charge for a pair and 40 bytes a clock it
// was 7 %: 300 x 10912 x 2048 SiLU gate 26.1 -> 18.2 us, 512 x 512 x 256 6.0 -> 4.8, 1000 x 1024 x 512 7.3 -> 6.1, 4096 x 3072 x 768 SwiGLU 20.9 either way.)
template <int EPI>
static int gemm_run(const GemmOperands& o, const GemmParams& p, int n_sm, int dev, cudaStream_t st) {
  const int n_kb = (p.K + kGK - 1) / kGK;
  int bn = 0, cg = 0;
  double best = 1e300;
  const int forms[7][2] = {{256, 2}, {192, 2}, {128, 2}, {256, 1}, {192, 1}, {128, 1}, {64, 1}};
  for (const auto& f : forms) {
    if (f[1] == 2 && p.M <= kGM) continue;  // half of the pair would have no rows
    const long long tiles = (long long)((p.M + f[1] * kGM - 1) / (f[1] * kGM)) * ((p.N + f[0] - 1) / f[0]);
    const long long slots = n_sm / f[1];
    const double block = fmax(2.0 * f[0], gemm_stage_bytes(f[0], f[1]) / 56.0);
    const double cost = (double)((tiles + slots - 1) / slots) * fmax(n_kb * block, 16.0 * f[0]) + (f[1] == 2 ? 4000.0 : 0.0);
    if (cost < best * 0.999) {
      best = cost;
      bn = f[0];
      cg = f[1];
    }
  }
  if (cg == 2) {
    if (bn == 256) return gemm_launch<256, 2, EPI>(o, p, n_sm, dev, st);
    if (bn == 192) return gemm_launch<192, 2, EPI>(o, p, n_sm, dev, st);
    return gemm_launch<128, 2, EPI>(o, p, n_sm, dev, st);
  }
  if (bn == 256) return gemm_launch<256, 1, EPI>(o, p, n_sm, dev, st);
  if (bn == 192) return gemm_launch<192, 1, EPI>(o, p, n_sm, dev, st);
  if (bn == 128) return gemm_launch<128, 1, EPI>(o, p, n_sm, dev, st);
  return gemm_launch<64, 1, EPI>(o, p, n_sm, dev, st);
}

}  // namespace tc
}  // namespace dgpt

using namespace dgpt;

extern "C" int dgpt_bounded_wait_probe(int32_t arrive, int64_t limit_cycles, int32_t* out, void* stream) {
  DGPT_REQUIRE(out, "bounded_wait_probe: NULL pointer");
  DGPT_REQUIRE(limit_cycles > 0 && limit_cycles <= 2000000000ll, "bounded_wait_probe: limit must be in (0, 2e9] cycles");
  tc::bounded_wait_probe_kernel<<<1, 64, 0, static_cast<cudaStream_t>(stream)>>>(arrive, limit_cycles, out);
  return launch_status("bounded_wait_probe");
}

int dgpt::linear_launch(const void* a, int64_t a_row_stride, const void* w, int64_t w_row_stride, void* out,
                        int64_t out_row_stride, const void* resid, int64_t resid_row_stride, int32_t M, int32_t N,
                        int32_t K, int32_t epilogue, float alpha, float limit, int32_t dtype, int32_t* status,
                        const HeadDraw* draw, bool tiles, void* stream) {
  DGPT_REQUIRE(a && w && (out || epilogue == 3), "linear: NULL pointer");
  DGPT_REQUIRE(M >= 0 && N > 0 && K > 0, "linear: bad sizes");
  DGPT_REQUIRE(epilogue >= 0 && epilogue <= 6,
               "linear: epilogue must be 0 (store), 1 (SwiGLU of interleaved pairs), 2 (add), 3 (draw), 4 (xIELU), 5 (SiLU gate) or 6 "
               "(soft-cap)");
  DGPT_REQUIRE(epilogue != 6 || alpha > 0.f, "linear: epilogue 6 needs a positive cap");
  DGPT_REQUIRE(epilogue != 2 || resid, "linear: epilogue 2 needs the matrix to add");
  DGPT_REQUIRE(epilogue != 3 || (draw && draw->best), "linear: epilogue 3 needs the draw parameters");
  if (dtype != DGPT_BF16) {
    set_error("linear: only bf16 is built (dtype %d)", dtype);
    return DGPT_E_UNSUPPORTED;
  }
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (!al(a) || !al(w) || (out && !al(out)) || K % 8 != 0 || N % 16 != 0 || a_row_stride % 8 != 0 || w_row_stride % 8 != 0 ||
      out_row_stride % 8 != 0 || (epilogue == 2 && (!al(resid) || resid_row_stride % 8 != 0))) {
    set_error("linear: pointers must be 16-byte aligned, K and the row strides multiples of 8, N a multiple of 16");
    return DGPT_E_UNSUPPORTED;
  }
  if (M == 0) return DGPT_OK;
  if (!tc::device_is_sm100() || tc::encode_fn() == nullptr) {
    set_error("linear: needs an sm_100 device and cuTensorMapEncodeTiled");
    return DGPT_E_UNSUPPORTED;
  }
  // The rows of W are read once either way, and nothing waits for tiles (16384 x 1024 in us: one row 13.0 -> 8.0, two 10.3, four 13.2).
  if (M <= kGemvMaxRows && epilogue != 3 && !tiles)
    return gemv_launch(a, a_row_stride, w, w_row_stride, out, out_row_stride, resid, resid_row_stride, M, N, K, epilogue, alpha, limit,
                       static_cast<cudaStream_t>(stream));
  static int n_sm[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    set_error("linear: cudaGetDevice failed");
    return DGPT_E_CUDA;
  }
  if (n_sm[dev] == 0) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n < 2) {
      set_error("linear: cudaDeviceGetAttribute failed");
      return DGPT_E_CUDA;
    }
    n_sm[dev] = n;
  }
  tc::GemmParams p;
  p.resid = static_cast<const __nv_bfloat16*>(resid);
  p.resid_rs = resid_row_stride;
  p.M = M; p.N = N; p.K = K;
  p.alpha = alpha; p.limit = limit;
  p.status = status;
  if (draw) p.draw = *draw;
  const tc::GemmOperands o{a, w, out, a_row_stride, w_row_stride, out_row_stride};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (epilogue) {
    case 0: return tc::gemm_run<0>(o, p, n_sm[dev], dev, st);
    case 1: return tc::gemm_run<1>(o, p, n_sm[dev], dev, st);
    case 2: return tc::gemm_run<2>(o, p, n_sm[dev], dev, st);
    case 3: return tc::gemm_run<3>(o, p, n_sm[dev], dev, st);
    case 4: return tc::gemm_run<4>(o, p, n_sm[dev], dev, st);
    case 5: return tc::gemm_run<5>(o, p, n_sm[dev], dev, st);
    default: return tc::gemm_run<6>(o, p, n_sm[dev], dev, st);
  }
}

extern "C" int dgpt_linear(const void* a, int64_t a_row_stride, const void* w, int64_t w_row_stride, void* out,
                           int64_t out_row_stride, const void* resid, int64_t resid_row_stride, int32_t M, int32_t N,
                           int32_t K, int32_t epilogue, float alpha, float limit, int32_t dtype, int32_t* status,
                           void* stream) {
  const bool tiles = epilogue >= 0 && (epilogue & DGPT_LINEAR_TILES) != 0;
  if (tiles) epilogue &= ~DGPT_LINEAR_TILES;
  DGPT_REQUIRE(epilogue >= 0 && epilogue <= 6 && epilogue != 3,
               "linear: epilogue must be 0 (store), 1 (SwiGLU of interleaved pairs), 2 (add), 4 (xIELU), 5 (SiLU gate) or 6 (soft-cap)");
  return linear_launch(a, a_row_stride, w, w_row_stride, out, out_row_stride, resid, resid_row_stride, M, N, K, epilogue, alpha,
                       limit, dtype, status, nullptr, tiles, stream);
}
