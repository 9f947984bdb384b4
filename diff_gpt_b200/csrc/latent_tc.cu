// Attention over cached rows on tcgen05 (sm_100a): one or two persistent CTAs per SM walk through (query row, head group,
// key split) items; the rows of an item pass through shared memory once and serve all its heads.
//
// A tile is 128 keys: dk columns of each row as keys and dv columns as values (the same columns where the cache holds
// latents), cut into units of 128 columns (two 64-column, 128-byte-swizzled blocks, 32 KB; one block where neither keys
// nor values have more than 64 columns).
//   S^T[key, head]    = K Q^T      M = 128 keys,    N = heads, K = dk    A: key units, K-major;            B: Q, K-major
//   O^T[column, head] += V^T P^T   M = 128 columns, N = heads, K = keys  A: a value unit, read MN-major;   B: P, K-major
// so the heads that share a row are the N of both products: 16, 32 or 64 of them cost the same passes over the tile, and
// nothing is padded to 128 rows of queries.  Decode is bound by reading the rows.
//   warp 5, lane 0  loader: Q of the item, then the units of its tiles into a ring, through TMA straight from the pages
//   warp 4, lane 0  issuer: S^T into one of two TMEM buffers, O^T += V^T P^T; with room in the ring the scores of the
//                   next tile are issued before the sums of this one
//   warps 0-3       softmax, one thread per key: probabilities against a running reference per head, kept in shared memory;
//                   when one of a row's is exceeded by 2^8 (found with one barrier vote per tile) all of that row's move to
//                   its maxima so far; written as bf16 into shared memory;
//                   after the item's last tile, one thread per column: normalise, gate, store
// Rows behind one prompt (ROWS): an item is a set of up to rg of them, whose heads together are the N of the products over
// the prompt's tiles; then come the tiles of each row's own slots (those of two rows in one tile where they fit its halves),
// whose products cover that row's columns only, so that a row with numbers that are none spoils no other (0 * NaN).  A product has 16 columns at
// least: rows with fewer heads (PACK) lie side by side for the prompt's tiles, and their sums move to 16 columns each before their own.  A row's result has the bits that it gets by itself, so that the tokens drawn from it do not depend on
// how many rows there are: a split is cut at the same tiles, references move row by row, and where a tile holds two rows' slots the second row's
// weights are handed to the threads that would have had them (tests/test_gpu_shared_rows.py).
// A row of a unit that holds fewer than 64 columns leaves the block's other accumulator rows undefined; they are not read.
// TMEM columns: S0 [0, N)  S1 [N, 2N)  O of unit u [2N + u N, +N)  PACK: O of unit u and row r [2N + UV N + 16 (u rg + r), +16).
// Every mbarrier wait is bounded.  When one runs out the abort flag is raised, the loader and the issuer stop and drain
// what they have in flight, the softmax warps run through their remaining tiles without waiting (so that every CTA
// barrier is still met by all of them), TMEM is freed and the status word names the wait.
#include "latent_attn.cuh"
#include "tcgen05.cuh"

namespace dgpt {
namespace tc {

constexpr int kLtKeys = 128;
constexpr uint32_t kLtBlock = kLtKeys * 128;  // [128 keys][64 columns] bf16, swizzled
constexpr uint32_t kLtUnit = 2 * kLtBlock;
constexpr int kLtThreads = 192;
constexpr int kLtMaxUnits = 10;

struct LtParams {
  LatentArgs a;
  int n_rows, n_groups, n_items;  // item = (split * n_sets + set) * n_groups + group
  int n_sets;                     // sets of rows: one row each, or
  int rg, cols, cols_log2;        // ROWS: up to rg rows of one prompt, each in `cols` columns: the heads that share a cache row, or 4 (latents: 16)
  int sets_per_prompt;
  int per, gpk;                   // heads that share a row, and item groups they make
  int n_units;                    // units in the ring
  uint32_t unit_bytes;
  int uk, uv, upt;                // units of a tile's keys and values (the same ones for latents), and of both
  int align;                      // tiles of a key range start at a multiple of this many slots
  int box;                        // slots per TMA box
};

// blocks of 64 columns in unit u of a vector of `cols` columns
__device__ __forceinline__ int lt_blocks(int cols, int u) { return cols - u * 128 > 64 ? 2 : 1; }

struct LtItem {
  int row, seq, g, h0, nh, split;
  int nr, n_shared;               // ROWS: rows of the set, tiles of their prompt
  int n_mine, own0, n_own;        // ROWS: this split's tiles of the prompt; its first tile of each row's own slots, and how many
  bool pairs;                     // own slots fit half a tile: one holds those of two rows
  int begin[3], end[3], base[3];  // the slot ranges and where their tiles start
  int n_first, n_second;          // tiles of the first range, of the first two
  int t0, n;                      // this split's tiles
};

// KEPT: the cache holds first keys that are seen from every distance, a slot range of their own
template <bool KEPT, bool ROWS>
__device__ __forceinline__ LtItem lt_item(const LtParams& p, int item, int N) {
  LtItem it;
  // Groups change fastest: those of a row lie beside each other in memory and are read at the same time, so DRAM pages are opened once.
  // 256 rows of 545 keys, 4 groups of 128: 83 -> 81 us, 200 rows of 1450, 8 groups: 236 -> 232.
  const int sp = item / p.n_groups, grp = item - sp * p.n_groups;
  it.split = sp / p.n_sets;
  it.row = sp - it.split * p.n_sets;
  it.nr = 1;
  if (ROWS) {
    const int prompt = it.row / p.sets_per_prompt, first = (it.row - prompt * p.sets_per_prompt) * p.rg;
    it.nr = min(p.rg, p.a.share - first);
    it.row = prompt * p.a.share + first;
  }
  it.g = 0;
  it.h0 = 0;
  int first = 0;
  if (p.n_groups > 1) {
    it.g = grp / p.gpk;
    first = (grp - it.g * p.gpk) * N;
    it.h0 = it.g * p.per + first;
  }
  it.nh = ROWS ? it.nr << p.cols_log2 : min(N, p.per - first);
  const LatentKeys k = latent_keys(p.a, it.row);
  it.seq = k.seq;
  // [0, ks) and [lo, n), cut where slots change from the first run to the second; the cut lies in one of the two
  const bool own = k.lo >= k.n0;
  it.begin[0] = 0;
  it.end[0] = KEPT ? min(k.ks, k.n0) : 0;
  it.begin[1] = own ? k.s1 : k.lo;
  it.end[1] = own ? (KEPT ? k.s1 + max(0, k.ks - k.n0) : k.s1) : k.n0;
  it.begin[2] = k.s1 + max(0, k.lo - k.n0);
  it.end[2] = k.s1 + (k.n - k.n0);
  int nt[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    it.base[i] = it.begin[i] & ~(p.align - 1);  // a power of two
    nt[i] = it.end[i] > it.begin[i] ? (it.end[i] - it.base[i] + kLtKeys - 1) / kLtKeys : 0;
  }
  it.n_first = KEPT ? nt[0] : 0;
  it.n_second = it.n_first + nt[1];
  it.n_shared = own ? it.n_first : it.n_second;
  // the tiles of one row, and those of them that are this split's
  const int total = it.n_second + nt[2];
  int t1 = total;
  it.t0 = 0;
  if (p.a.n_splits > 1) {
    const int per = (total + p.a.n_splits - 1) / p.a.n_splits;
    it.t0 = min(total, it.split * per);
    t1 = min(total, it.t0 + per);
  }
  it.n = t1 - it.t0;
  it.pairs = false;
  if (ROWS) {
    it.n_mine = max(0, min(t1, it.n_shared) - it.t0);
    it.own0 = max(it.t0, it.n_shared);
    it.n_own = max(0, t1 - it.own0);
    it.pairs = p.box <= kLtKeys / 2 && total - it.n_shared == 1 && nt[2] == 1 && it.end[2] - it.base[2] <= kLtKeys / 2;
    it.n = it.n_mine + (it.pairs ? (it.nr + 1) / 2 * it.n_own : it.nr * it.n_own);
  }
  return it;
}
struct LtTile {
  int slot, begin, end;  // first slot; the limits of the slots that are seen
  int own;               // the row of the set whose slots they are, -1: those of all
  bool pair;             // the second half of the tile: the same slots of the next row
};
template <bool KEPT, bool ROWS>
__device__ __forceinline__ LtTile lt_tile(const LtItem& it, int j) {
  LtTile x;
  int t = it.t0 + j;
  x.own = -1;
  x.pair = false;
  if (ROWS && j >= it.n_mine) {
    t = j - it.n_mine;
    x.pair = it.pairs;
    x.own = it.pairs ? 2 * t : t / it.n_own;
    t = it.own0 + (it.pairs ? 0 : t - x.own * it.n_own);
  }
  if (KEPT && t < it.n_first) {
    x.begin = it.begin[0];
    x.end = it.end[0];
    x.slot = it.base[0] + t * kLtKeys;
    return x;
  }
  const bool last = t >= it.n_second;
  x.begin = last ? it.begin[2] : it.begin[1];
  x.end = last ? it.end[2] : it.end[1];
  x.slot = (last ? it.base[2] : it.base[1]) + (t - (last ? it.n_second : it.n_first)) * kLtKeys;
  return x;
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// The four softmax warps: a barrier, and a barrier that tells every thread whether any of them said yes.
__device__ __forceinline__ void lt_sync() { asm volatile("barrier.sync 1, 128;" ::: "memory"); }
__device__ __forceinline__ bool lt_any(bool mine) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbarrier.red.or.pred q, 2, 128, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((int)mine)
      : "memory");
  return r != 0;
}
// op over the 32 lanes for each of 16 values at once: lane l returns the result of value l & 15.  Every step halves the
// values a lane still carries, so 16 shuffles do the work of 80.
template <typename F>
__device__ __forceinline__ float lt_reduce16(const float* v, int lane, F op) {
  float a[8], b[4], c[2];
#pragma unroll
  for (int i = 0; i < 8; ++i) {  // keep values 8 (lane bit 3) + i
    const bool hi = lane & 8;
    const float keep = hi ? v[8 + i] : v[i], send = hi ? v[i] : v[8 + i];
    a[i] = op(keep, __shfl_xor_sync(0xffffffffu, send, 8));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool hi = lane & 4;
    const float keep = hi ? a[4 + i] : a[i], send = hi ? a[i] : a[4 + i];
    b[i] = op(keep, __shfl_xor_sync(0xffffffffu, send, 4));
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const bool hi = lane & 2;
    const float keep = hi ? b[2 + i] : b[i], send = hi ? b[i] : b[2 + i];
    c[i] = op(keep, __shfl_xor_sync(0xffffffffu, send, 2));
  }
  const bool hi = lane & 1;
  const float keep = hi ? c[1] : c[0], send = hi ? c[0] : c[1];
  const float d = op(keep, __shfl_xor_sync(0xffffffffu, send, 1));
  return op(d, __shfl_xor_sync(0xffffffffu, d, 16));
}

// NB: columns of the products = 16 NB; HS <= 16 NB: heads the softmax looks after (a group may hold fewer than 16).
// SHARED: a tile's values are its keys (latents), whose cache has no kept first keys.
// ROWS: a column is a head of one of rg rows, column c = row c >> cols_log2, head c & (cols - 1); HS = min(cols, 16).
template <int NB, int HS, bool SHARED, bool ROWS>
__global__ void __launch_bounds__(kLtThreads, NB == 4 ? 1 : 2)
latent_tc_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mc, const LtParams p) {
  constexpr int N = 16 * NB, CW = ROWS ? N : HS;  // columns, and those that the softmax looks after
  constexpr bool PACK = ROWS && HS < 16;
  // The sums of a tile that is not full go over the 16-key steps that hold a key only.  Latents of 512 / 256, 256 rows with
  // 1000 keys: 106.5 -> 102.4 and 36.9 -> 33.8 us.  Rows of keys and values, each by itself, have products to spare (they
  // wait for HBM) and took longer with them issued one by one: 64.3 -> 66.5 (4 groups of 64), 235 -> 241 (8 of 128).
  constexpr bool kSome = SHARED || ROWS;
  constexpr uint32_t kIdescS = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | (8u << 24);
  constexpr uint32_t kIdescO = kIdescS | (1u << 15);  // A is read MN-major
  constexpr uint32_t kQBlock = N * 128;               // [N heads][64 columns]
  constexpr uint32_t kPBlock = N * 128;               // [N heads][64 keys]
  constexpr uint32_t kTmemCols = NB == 1 ? 128 : (NB == 2 ? 256 : 512);  // N (2 + 4) columns at most; PACK: as lt_rows allows
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int UT = p.upt, UK = p.uk, UV = p.uv, NU = p.n_units;
  const int v_unit = SHARED ? 0 : UK;  // where a tile's value units start
  const int nqb = SHARED ? 2 * UK : (p.a.dk + 63) / 64;  // 64-column blocks of Q
  const uint32_t unit_bytes = SHARED ? kLtUnit : p.unit_bytes;
  uint8_t* sU = smem;
  uint8_t* sQ = sU + (size_t)NU * unit_bytes;
  uint8_t* sP = sQ + (size_t)2 * UK * kQBlock;  // one or two buffers of two blocks
  // With room in the ring for the next tile's keys beside a tile the scores of the next tile are issued before the sums
  // of this one, and P needs two buffers; otherwise the next scores follow the sums, and their arrival also says that P has been read.  (Issuing
  // the part of the next scores that the ring could hold before the sums was measured 12 % slower: every change between
  // the two kinds of product costs the tensor pipe more than the wait it fills.)
  const bool ahead = NU >= UT + UK;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sP + (ahead ? 4 : 2) * kPBlock);
  float* red = reinterpret_cast<float*>(bars + 32);  // [4 warps][N]
  float* fac = red + 4 * N;                          // [4 warps][N]
  float* ref = fac + 4 * N;                          // [N] what the probabilities of a head are relative to
  float* hand = ref + N;                             // ROWS, half tiles: [N / 2][64 keys] weights of second rows
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ROWS && p.box <= kLtKeys / 2 ? hand + 32 * N : hand);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t aU = smem_u32(sU), aQ = smem_u32(sQ), aP = smem_u32(sP);
  const uint32_t bar0 = smem_u32(bars);
  const uint32_t bar_q = bar0, bar_qf = bar0 + 8, bar_of = bar0 + 16, bar_drain = bar0 + 24, bar_s = bar0 + 32, bar_p = bar0 + 48,
                 bar_o = bar0 + 64, bar_u = bar0 + 80, bar_uf = bar_u + 8 * kLtMaxUnits;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 10 + 2 * kLtMaxUnits; ++i) mbar_init(bar0 + 8 * i, (i == 2 || i == 6 || i == 7) ? 128 : 1);  // O free; P ready
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  dep_begin();

  if (warp == 5) {
    // ================= loader =================
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mq)) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mc)) : "memory");
      unsigned un = 0u, items = 0u;  // units and items loaded so far
      bool ok = true;
      const int pt = p.a.kv.page_tokens;
      const LatentArgs& a = p.a;
      for (int item = blockIdx.x; ok && item < p.n_items; item += gridDim.x) {
        const LtItem it = lt_item<!SHARED, ROWS>(p, item, N);
        if (it.n == 0) continue;
        if (items > 0) ok = wait_or_abort(bar_qf, (items - 1) & 1u, abort_flag, 50);  // the last scores of the item before are done
        if (!ok) break;
        mbar_expect_tx(bar_q, (uint32_t)nqb * kQBlock);
        for (int c = 0; c < nqb; ++c) tma_load_3d(aQ + c * kQBlock, &mq, bar_q, c * 64, it.h0, it.row);
        ++items;
        for (int j = 0; ok && j < it.n; ++j) {
          const LtTile x = lt_tile<!SHARED, ROWS>(it, j);
          const int seq0 = it.seq + (ROWS ? max(x.own, 0) : 0);
          const int half = min(kLtKeys / p.box, (x.end - x.slot + p.box - 1) / p.box);  // boxes of a row
          const int boxes = ROWS && x.pair && x.own + 1 < it.nr ? 2 * half : half;
          for (int u = 0; ok && u < UT; ++u, ++un) {
            const unsigned s = un % (unsigned)NU, round = un / (unsigned)NU;
            if (round > 0) ok = wait_or_abort(bar_uf + 8 * s, (round - 1) & 1u, abort_flag, 51);
            if (!ok) break;
            const uint32_t full = bar_u + 8 * s, dst = aU + s * unit_bytes;
            const bool key = u < UK;
            const int blocks = SHARED ? 2 : key ? lt_blocks(a.dk, u) : lt_blocks(a.dv, u - UK);
            const int col = SHARED ? u * 128 : key ? it.g * a.dk + u * 128 : a.v_col + it.g * a.dv + (u - UK) * 128;
            mbar_expect_tx(full, (uint32_t)boxes * p.box * 128u * blocks);
            for (int b = 0; b < boxes; ++b) {
              const bool second = ROWS && b >= half;
              const int seq = seq0 + (second ? 1 : 0), at = x.slot + (second ? b - half : b) * p.box;
              const uint32_t to = dst + (second ? kLtBlock / 2 + (b - half) * p.box * 128 : b * p.box * 128);
              int pg = seq, in = at;
              if (p.a.kv.page_table) {
                const int lp = at / pt;
                pg = p.a.kv.page_table[(long long)seq * p.a.kv.max_pages + lp];
                in = at - lp * pt;
              }
              tma_load_3d(to, &mc, full, col, in, pg);
              if (blocks == 2) tma_load_3d(to + kLtBlock, &mc, full, col + 64, in, pg);
            }
          }
        }
      }
      if (!ok || *abort_flag) {  // let the copies in flight land
        if (p.a.status) atomicExch(p.a.status, *abort_flag ? *abort_flag : 50);
        if (items > 0) mbar_wait(bar_q, (items - 1) & 1u);
        for (unsigned i = 0; i < (unsigned)NU && i < un; ++i)
          mbar_wait(bar_u + 8 * ((un - 1 - i) % (unsigned)NU), ((un - 1 - i) / (unsigned)NU) & 1u);
      }
    }
  } else if (warp == 4) {
    // ================= MMA issuer =================
    if (lane == 0) {
      const uint64_t dC = smem_desc(0, 16, 1024), dM = smem_desc(0, kLtBlock, 1024);  // K-major rows; MN-major pairs of blocks
      // the products of rows' own slots: of their columns only
      auto own_n = [&](const LtTile& x, uint32_t idesc, int rows) {
        return !ROWS || x.own < 0 ? idesc : (idesc & ~(63u << 17)) | (uint32_t)max(2, rows * p.cols >> 3) << 17;
      };
      auto own_block = [&](const LtTile& x) { return ROWS && x.own >= 0 ? (x.own << p.cols_log2) >> 4 : 0; };
      unsigned g = 0u, items = 0u;  // tiles; items
      bool ok = true;
      for (int item = blockIdx.x; ok && item < p.n_items; item += gridDim.x) {
        const LtItem it = lt_item<!SHARED, ROWS>(p, item, N);
        if (it.n == 0) continue;
        ok = wait_or_abort(bar_q, items & 1u, abort_flag, 52);
        unsigned started = 0u;  // 16-column blocks of O that hold sums; PACK: from bit 4 on those of the rows
        auto issue_s = [&](unsigned gt, int j) {
          const bool last = j + 1 == it.n;
          const LtTile x = lt_tile<!SHARED, ROWS>(it, j);
          const int blk = own_block(x);
          const uint32_t idesc = own_n(x, kIdescS, x.pair ? 2 : 1);
          const uint32_t d = tmem + (gt & 1u) * N + blk * 16;
          for (int u = 0; ok && u < UK; ++u) {
            const unsigned un = gt * (unsigned)UT + (unsigned)u, s = un % (unsigned)NU;
            ok = wait_or_abort(bar_u + 8 * s, (un / (unsigned)NU) & 1u, abort_flag, 53);
            if (!ok) return;
            tc_fence_after();
            const uint64_t da = dC + ((aU + s * unit_bytes) >> 4), db = dC + ((aQ + 2 * u * kQBlock + blk * 2048) >> 4);
            if (SHARED || lt_blocks(p.a.dk, u) == 2) umma_ss8<2, kLtBlock / 16, 2, kQBlock / 16>(d, da, db, idesc, u > 0 ? 1u : 0u);
            else umma_ss4<2, 2>(d, da, db, idesc, u > 0 ? 1u : 0u);
            if (!SHARED) umma_commit(bar_uf + 8 * s);  // keys are done with
          }
          umma_commit(bar_s + 8 * (gt & 1u));
          if (last) umma_commit(bar_qf);
        };
        if (ok) issue_s(g, 0);
        for (int j = 0; ok && j < it.n; ++j, ++g) {
          const unsigned b = g & 1u;
          if (ahead && j + 1 < it.n) issue_s(g + 1, j + 1);
          ok = ok && wait_or_abort(bar_p + 8 * b, (g >> 1) & 1u, abort_flag, 54);
          if (ok && j == 0 && items > 0) ok = wait_or_abort(bar_of, (items - 1) & 1u, abort_flag, 55);  // the last item's O has been read
          if (!ok) break;
          tc_fence_after();
          const LtTile x = lt_tile<!SHARED, ROWS>(it, j);
          // steps of 16 keys that hold one that is seen: the others' probabilities are zeros
          const int k0 = kSome ? max(x.begin - x.slot, 0) >> 4 : 0, k1 = kSome ? min(kLtKeys, x.end - x.slot + 15) >> 4 : 8;
          const bool apart = PACK && x.own >= 0;  // sums in the row's own 16 columns, P in the first 16 rows of its buffer
          const int blk = apart ? 0 : own_block(x), bit = apart ? 4 + x.own : blk;
          const uint32_t idesc = own_n(x, kIdescO, 1);
          const bool second = ROWS && x.pair && x.own + 1 < it.nr;
          const int more = PACK ? 1 : p.cols >> 4;  // from a row's blocks to the next row's
          if (PACK && x.own >= 0 && it.n_mine > 0) started = ~0u;  // the prompt's sums have been moved there
          const unsigned acc = (started >> bit) & 1u, acc2 = (started >> (bit + more)) & 1u;
          started |= ROWS && x.own >= 0 ? (1u << bit) | (second ? 1u << (bit + more) : 0u) : 15u;  // a row's own blocks are always touched together
          for (int u = 0; u < UV; ++u) {
            const unsigned un = g * (unsigned)UT + (unsigned)(v_unit + u), s = un % (unsigned)NU;
            if (!SHARED) {
              ok = wait_or_abort(bar_u + 8 * s, (un / (unsigned)NU) & 1u, abort_flag, 53);
              if (!ok) break;
              tc_fence_after();
            }
            const uint32_t d = tmem + (apart ? 2 * N + UV * N + (u * p.rg + x.own) * 16 : 2 * N + u * N + blk * 16);
            const uint64_t da = dM + ((aU + s * unit_bytes) >> 4), db = dC + ((aP + (ahead ? 2 * b * kPBlock : 0u) + blk * 2048) >> 4);
            if (k0 == 0 && k1 == 8) umma_ss8<128, 512, 2, kPBlock / 16>(d, da, db, idesc, acc);
            else {
              for (int k = k0; k < k1; ++k) umma_ss(d, da + 128 * k, db + (k >> 2) * (kPBlock / 16) + 2 * (k & 3), idesc, k > k0 ? 1u : acc);
              if (second)
                for (int k = k0; k < k1; ++k)
                  umma_ss(d + 16 * more, da + 512 + 128 * k, db + kPBlock / 16 + (PACK ? 0 : 128 * more) + 2 * k, idesc, k > k0 ? 1u : acc2);
            }
            umma_commit(bar_uf + 8 * s);
          }
          if (!ok) break;
          umma_commit(bar_o + 8 * b);
          if (!ahead && j + 1 < it.n) issue_s(g + 1, j + 1);
        }
        ++items;
      }
      if (!ok || *abort_flag) {
        if (p.a.status) atomicExch(p.a.status, *abort_flag ? *abort_flag : 52);
        umma_commit(bar_drain);  // completes when everything issued so far has finished
        mbar_wait(bar_drain, 0);
      }
    }
  } else {
    // ================= softmax: one thread per key; one thread per column at the end =================
    const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
    unsigned g = 0u;
    bool fail = false;
    const long long RH = (long long)p.n_rows * p.a.H;
    if (CW < N)  // heads nobody looks after: their probabilities are zeros, once
      for (int i = tid; i < (int)((ahead ? 4 : 2) * kPBlock / 16); i += 128) reinterpret_cast<uint4*>(sP)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid < N) ref[tid] = -INFINITY;
    lt_sync();
    auto row_of = [&](int c) -> long long { return ROWS ? c >> p.cols_log2 : 0; };
    auto head_of = [&](int c) -> long long { return ROWS ? c & (p.cols - 1) : c; };
    auto there = [&](int c, int nh) { return c < nh && (!ROWS || head_of(c) < p.per); };  // the column is a head's
    for (int item = blockIdx.x; item < p.n_items; item += gridDim.x) {
      const LtItem it = lt_item<!SHARED, ROWS>(p, item, N);
      const int nh = it.nh;
      unsigned started = 0u;  // 16-column blocks of O that hold sums; PACK: from bit 4 on those of the rows
      constexpr int HL = (N + 31) / 32;  // heads a lane looks after at the end of the item
      float gate[HL];
#pragma unroll
      for (int c = 0; c < HL; ++c) {  // wanted at the end only
        const int h = lane + 32 * c;
        gate[c] = 1.f;
        if (p.a.gate && there(h, nh))
          gate[c] = __bfloat162float(static_cast<const __nv_bfloat16*>(p.a.gate)[(it.row + row_of(h)) * p.a.gate_rs + it.h0 + head_of(h)]);
      }
      float l[CW];
#pragma unroll
      for (int h = 0; h < CW; ++h) l[h] = 0.f;
      for (int j = 0; j < it.n; ++j, ++g) {
        const unsigned b = g & 1u;
        const LtTile x = lt_tile<!SHARED, ROWS>(it, j);
        const int half = ROWS && x.pair ? tid >> 6 : 0, slot = x.slot + tid - 64 * half, end = x.end;
        // The tile concerns columns [c_lo, c_hi), this thread's key [k_lo, k_hi) of them.
        const int c_lo = ROWS && x.own >= 0 ? x.own << p.cols_log2 : 0;
        const int c_hi = ROWS && x.own >= 0 ? c_lo + (x.pair ? 2 : 1) * p.cols : CW;
        const int k_lo = c_lo + half * p.cols, k_hi = ROWS && x.own >= 0 ? k_lo + p.cols : CW;
        auto block = [&](int c) { return !ROWS || (c_lo < 16 * c + 16 && c_hi > 16 * c); };
        const bool seen = slot >= x.begin && slot < end && (!ROWS || x.own + half < it.nr);
        auto columns = [&](int c) -> unsigned {  // of block c, one bit each
          if (!seen) return 0u;
          if (ROWS && x.own < 0) return 0xffffu;
          const int lo = max(k_lo - 16 * c, 0), hi = min(k_hi - 16 * c, 16);
          return hi > lo ? (1u << hi) - (1u << lo) : 0u;
        };
        if (!fail && !wait_or_abort(bar_s + 8 * b, (g >> 1) & 1u, abort_flag, 56)) fail = true;
        fail = __any_sync(0xffffffffu, fail);
        tc_fence_after();
        // Nothing was loaded here, or rows nobody has written: 0 * x must stay 0 where the sums go over the slot.  The whole warp
        // waits for the unit: lanes that go apart in a wait need not have met again at the loads and barriers that follow, which
        // are the warp's.
        const bool blank = slot >= end && (!kSome || slot - x.slot < ((end - x.slot + 15) & ~15));
        if (!fail && __any_sync(0xffffffffu, blank)) {
          for (int u = 0; u < UV; ++u) {
            const unsigned un = g * (unsigned)UT + (unsigned)(v_unit + u), us = un % (unsigned)NU;
            if (!SHARED && !wait_or_abort(bar_u + 8 * us, (un / (unsigned)NU) & 1u, abort_flag, 59)) break;  // still on its way
            uint8_t* unit = sU + (size_t)us * unit_bytes;
            const bool two = SHARED || lt_blocks(p.a.dv, u) == 2;
            if (blank) {
#pragma unroll
              for (int c = 0; c < 8; ++c) {
                reinterpret_cast<uint4*>(unit + tid * 128)[c] = make_uint4(0u, 0u, 0u, 0u);
                if (two) reinterpret_cast<uint4*>(unit + kLtBlock + tid * 128)[c] = make_uint4(0u, 0u, 0u, 0u);
              }
            }
          }
        }
        __syncwarp();
        // the rows' columns in O, and whether a product on them may be in flight or done
        auto rows_at = [&](int u, int r) { return lane_addr + 2 * N + UV * N + (u * p.rg + r) * 16; };
        const bool apart = PACK && x.own >= 0;
        if (apart && it.n_mine > 0 && started < 16u) {  // the prompt's sums move to the rows' own columns
          if (!fail && !wait_or_abort(bar_o + 8 * (b ^ 1u), ((g - 1) >> 1) & 1u, abort_flag, 57)) fail = true;
          fail = __any_sync(0xffffffffu, fail);
          tc_fence_after();
#pragma unroll 1
          for (int i = 0; i < UV * NB; ++i) {
            const int u = i / NB, c = i - u * NB;
            float v[16];
            tmem_ld16_nowait(lane_addr + 2 * N + u * N + c * 16, v);
            tc_wait_ld();
#pragma unroll
            for (int q = 0; q < 16 / HS; ++q) {
              uint32_t w[16];
#pragma unroll
              for (int k = 0; k < 16; ++k) w[k] = k < HS ? __float_as_uint(v[(q * HS + k) % 16]) : 0u;
              tmem_st16(rows_at(u, c * (16 / HS) + q), w);
            }
          }
          tc_wait_st();
          started = ~0u;
        }
        float s[N];  // log2 of what is added for this key, against the heads' references (a score is rounded before its reference is taken off)
        for (int pass = 0;; ++pass) {
#pragma unroll
          for (int c = 0; c < NB; ++c) tmem_ld16_nowait(lane_addr + b * N + c * 16, s + 16 * c);
          tc_wait_ld();
          float top = -INFINITY;
#pragma unroll
          for (int c = 0; c < NB; ++c) {
            if (!block(c)) continue;
            const unsigned cols = columns(c);
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              if (16 * c + i >= CW) continue;
              const float4 m4 = *reinterpret_cast<const float4*>(ref + 16 * c + i);
              const float mm[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const int h = 16 * c + i + k;
                s[h] = (cols >> (i + k)) & 1u ? __fmul_rn(s[h], p.a.scale_log2) - mm[k] : -INFINITY;
                top = fmaxf(top, s[h]);
              }
            }
          }
          if (pass || !lt_any(top >= 8.f && !fail)) break;  // (a score above the rounded reference + 8 is 8 above the reference)
          // Some row's references have to move.  Rare but for an item's first tile, so the loops stay rolled: with every
          // block's code laid out the instructions of a first tile took longer to fetch than the tile.
#pragma unroll 1
          for (int c = c_lo >> 4; c < NB && 16 * c < c_hi; ++c) {
            float v[16];
            tmem_ld16_nowait(lane_addr + b * N + c * 16, v);
            tc_wait_ld();
            const unsigned cols = columns(c);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = (cols >> i) & 1u ? __fmul_rn(v[i], p.a.scale_log2) : -INFINITY;
            const float t = lt_reduce16(v, lane, [](float x, float y) { return fmaxf(x, y); });
            if (lane < 16) red[warp * N + 16 * c + lane] = t;
          }
          lt_sync();
          if (warp < (N + 31) / 32) {
            const bool in = tid >= c_lo && tid < c_hi;  // (c_hi <= N)
            const float mo = in ? ref[tid] : 0.f;
            const float mt = in ? fmaxf(fmaxf(red[tid], red[N + tid]), fmaxf(red[2 * N + tid], red[3 * N + tid])) : 0.f;
            const unsigned want = __ballot_sync(0xffffffffu, in && mt > mo + 8.f);
            // rows together: those of the row in whose columns one wants to (there are at most 32 of them, within the warp)
            const bool move = in && (!ROWS || (want >> (lane & ~(p.cols - 1)) & (p.cols == 32 ? ~0u : (1u << p.cols) - 1u)) != 0u);
            float alpha = 1.f;
            if (move) {
              const float mn = fmaxf(mt, mo);
              alpha = mn == -INFINITY ? 1.f : ex2(mo - mn);  // -inf before the first tile: 0
              ref[tid] = mn;
            }
            if (tid < N) fac[tid] = alpha;
          }
          __syncwarp();
          lt_sync();  // and `red` may be written again
#pragma unroll
          for (int h = 0; h < CW; h += 4) {
            const float4 f = *reinterpret_cast<const float4*>(fac + h);
            l[h] *= f.x;
            l[h + 1] *= f.y;
            l[h + 2] *= f.z;
            l[h + 3] *= f.w;
          }
          if (apart ? (started >> (4 + x.own)) & 3u : started) {
            // O may only be touched when no product is in flight on it: the tile before must be done, and this tile's
            // waits for this thread's arrival below
            if (!fail && !wait_or_abort(bar_o + 8 * (b ^ 1u), ((g - 1) >> 1) & 1u, abort_flag, 57)) fail = true;
            fail = __any_sync(0xffffffffu, fail);
            tc_fence_after();
            if (apart) {
#pragma unroll 1
              for (int i = 0; i < UV * (x.pair ? 2 : 1); ++i) {
                const int u = i % UV, r = x.own + i / UV;
                if (!((started >> (4 + r)) & 1u)) continue;
                float v[16];
                tmem_ld16_nowait(rows_at(u, r), v);
                tc_wait_ld();
                uint32_t w[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) w[k] = k < HS ? __float_as_uint(v[k] * fac[r * HS + k]) : 0u;
                tmem_st16(rows_at(u, r), w);
              }
            } else
#pragma unroll 1
            for (int c = c_lo >> 4; c < NB && 16 * c < c_hi; ++c) {
              if (!((started >> c) & 1u)) continue;
#pragma unroll 1
              for (int u = 0; u < UV; ++u) {
                float v[16];
                const uint32_t addr = lane_addr + 2 * N + u * N + c * 16;
                tmem_ld16_nowait(addr, v);
                tc_wait_ld();
                uint32_t w[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(v[i] * fac[16 * c + i]);
                tmem_st16(addr, w);
              }
            }
            tc_wait_st();
          }
        }
        uint8_t* pb = sP + ((ahead ? 2 * b : 0u) + (tid >> 6)) * kPBlock + (tid & 7) * 2;
        const int chunk = (tid & 63) >> 3;
        const float mine = half ? 0.f : 1.f;
#pragma unroll
        for (int c = 0; c < NB; ++c) {
          if (!block(c)) continue;
          if (!apart) started |= 1u << c;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int h = 16 * c + i;
            if (h >= CW) continue;
            s[h] = ex2(s[h]);  // not seen: 0
            l[h % CW] = ROWS ? fmaf(s[h], mine, l[h % CW]) : l[h % CW] + s[h];
            if (!apart) *reinterpret_cast<__nv_bfloat16*>(pb + h * 128 + ((chunk ^ (h & 7)) << 4)) = __float2bfloat16_rn(s[h]);
          }
          if (apart) {  // one block: the row's columns first
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int at = (i - k_lo) & 15;
              *reinterpret_cast<__nv_bfloat16*>(pb + at * 128 + ((chunk ^ (at & 7)) << 4)) = __float2bfloat16_rn(s[(16 * c + i) % N]);
            }
          }
        }
        if (apart) started |= (x.pair ? 3u : 1u) << (4 + x.own);
        fence_async_smem();
        tc_fence_before();
        mbar_arrive(bar_p + 8 * b);
        if (ROWS && half && x.own + 1 < it.nr) {  // the second row of a tile: its weights are summed by the threads that would have had them were it by itself
          float* to = hand + (x.own >> 1) * p.cols * 64 + (tid & 63);
#pragma unroll
          for (int c = 0; c < NB; ++c) {
            if (!block(c)) continue;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int j = 16 * c + i - k_lo;
              if (j >= 0 && j < p.cols) to[j * 64] = s[(16 * c + i) % N];
            }
          }
        }
      }
      // ---- the item's result ----
      if (it.n > 0) {
        const unsigned last = g - 1u;
        if (!fail && !wait_or_abort(bar_o + 8 * (last & 1u), (last >> 1) & 1u, abort_flag, 58)) fail = true;
        fail = __any_sync(0xffffffffu, fail);
        tc_fence_after();
      }
      if (ROWS && it.pairs && it.n_own > 0) {
        lt_sync();
        if (tid < 64) {
#pragma unroll
          for (int h = 4; h < CW; h += 4) {  // (a row's columns are four or more)
            const int r = h >> p.cols_log2;
            if (!(r & 1) || h >= nh) continue;
            const float* from = hand + ((r >> 1 << p.cols_log2) + (h & (p.cols - 1))) * 64 + tid;
#pragma unroll
            for (int i = 0; i < 4; ++i) l[h + i] += from[64 * i];
          }
        }
      }
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        float ls[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) ls[i] = 16 * c + i < CW ? l[(16 * c + i) % CW] : 0.f;
        const float t = lt_reduce16(ls, lane, [](float x, float y) { return x + y; });
        if (lane < 16) red[warp * N + 16 * c + lane] = t;
      }
      lt_sync();
      // where column c's parts go
      auto part = [&](int c) { return (long long)it.split * RH + (it.row + row_of(c)) * p.a.H + it.h0 + head_of(c); };
      // lane h: 1 / sum and gate of head h, or the sum itself for a split
#pragma unroll
      for (int c = 0; c < HL; ++c) {
        const int h = lane + 32 * c;
        if (h < N) {
          const float sum = (red[h] + red[N + h]) + (red[2 * N + h] + red[3 * N + h]);
          float f = sum > 0.f ? 1.f / sum : 0.f;
          if (p.a.gate) f *= 1.f / (1.f + __expf(-gate[c]));
          fac[warp * N + h] = f;
          if (p.a.n_splits > 1 && warp == 0 && there(h, nh)) {
            p.a.ws_ml[2 * part(h)] = ref[h];
            p.a.ws_ml[2 * part(h) + 1] = sum;
          }
          if (warp == 0) ref[h] = -INFINITY;
        }
      }
      lt_sync();  // `red` may be written again, `fac` is complete
      if (it.n > 0) {
#pragma unroll 1
        for (int u = 0; u < UV; ++u) {
          const int col = u * 128 + tid;
#pragma unroll 1
          for (int c = 0; c < NB; ++c) {
            float v[16];
            if (PACK && it.n_own > 0) {
#pragma unroll
              for (int q = 0; q < 16 / HS; ++q) {
                float t[16];
                tmem_ld16_nowait(lane_addr + 2 * N + UV * N + (u * p.rg + c * (16 / HS) + q) * 16, t);
                tc_wait_ld();
#pragma unroll
                for (int k = 0; k < HS; ++k) v[(q * HS + k) % 16] = t[k];
              }
            } else {
              tmem_ld16_nowait(lane_addr + 2 * N + u * N + c * 16, v);
              tc_wait_ld();
            }
            if (u == UV - 1 && c == NB - 1) {
              tc_fence_before();
              mbar_arrive(bar_of);  // the next item may overwrite O
            }
            if (p.a.n_splits > 1) {
              if (col < p.a.dv) {
#pragma unroll
                for (int i = 0; i < 16; ++i)
                  if (there(16 * c + i, nh)) p.a.ws_o[part(16 * c + i) * p.a.dv + col] = v[i];
              }
              continue;
            }
            // two columns of one head per store: an even lane takes the even head of a pair, its neighbour the odd one
            // (dv is a multiple of 8, so both columns exist or neither does)
            const bool odd = lane & 1;
            __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.a.out) + (long long)it.row * p.a.out_rs + (long long)it.h0 * p.a.dv + (col & ~1);
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              const float x = v[i] * fac[warp * N + 16 * c + i], y = v[i + 1] * fac[warp * N + 16 * c + i + 1];
              const float got = __shfl_xor_sync(0xffffffffu, odd ? x : y, 1);
              const int h = 16 * c + i + (odd ? 1 : 0);
              if (there(h, nh) && col < p.a.dv)
                *reinterpret_cast<__nv_bfloat162*>(dst + row_of(h) * p.a.out_rs + head_of(h) * p.a.dv) = odd ? __floats2bfloat162_rn(got, y) : __floats2bfloat162_rn(x, got);
            }
          }
        }
      } else if (p.a.n_splits == 1) {  // no keys at all
        for (int u = 0; u < UV; ++u) {
          const int col = u * 128 + tid;
          for (int h = 0; h < nh && col < p.a.dv; ++h)
            if (there(h, nh)) static_cast<__nv_bfloat16*>(p.a.out)[(it.row + row_of(h)) * p.a.out_rs + (it.h0 + head_of(h)) * p.a.dv + col] = __float2bfloat16_rn(0.f);
        }
      }
    }
    if (fail && p.a.status && tid == 0) atomicExch(p.a.status, *abort_flag ? *abort_flag : 56);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

static bool encode_3d(CUtensorMap* map, const void* base, const cuuint64_t (&dims)[3], const cuuint64_t (&strides)[2],
                      const cuuint32_t (&box)[3]) {
  const cuuint32_t ones[3] = {1, 1, 1};
  CUresult r = encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, ones,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("latent_attn: cuTensorMapEncodeTiled failed with %d", (int)r);
    return false;
  }
  return true;
}

// heads per group (per = heads that share a row), and what fits beside Q and P in the shared memory (limit: opt-in bytes per CTA)
static int lt_heads(int per) { return per <= 16 ? 16 : (per <= 32 ? 32 : 64); }
// columns that a row has where rows are taken together: as many as the softmax looks after where the row is by itself, since all its references move
// when any of them is exceeded, the other groups' heads among them
static int lt_cols(const LatentArgs& a) {
  const int per = a.H / a.G;
  return a.v_col == 0 ? (per < 16 ? 16 : per) : per < 4 ? 4 : per;
}
struct LtShape {
  int N, uk, uv, upt, hand;
  uint32_t unit_bytes;
  size_t bytes(int units) const {
    return (size_t)2 * uk * N * 128 + (size_t)(units >= upt + uk ? 4 : 2) * N * 128 + 256 + (size_t)36 * N + hand + 64 + 1024 + (size_t)units * unit_bytes +
           (unit_bytes < kLtUnit ? kLtBlock : 0);  // a value unit of one block is read as a pair of blocks: the last one's partner must exist
  }
  int units(size_t limit) const {
    int n = kLtMaxUnits;
    while (n > 0 && bytes(n) > limit) --n;
    return n;
  }
};
static LtShape lt_shape(const LatentArgs& a, int rows) {
  LtShape s;
  s.N = lt_heads(rows > 1 ? lt_cols(a) * rows : a.H / a.G);
  s.hand = rows > 1 && a.kv.page_tokens <= kLtKeys / 2 ? s.N * 128 : 0;
  s.uk = (a.dk + 127) / 128;
  s.uv = (a.dv + 127) / 128;
  s.upt = a.v_col == 0 ? s.uk : s.uk + s.uv;
  s.unit_bytes = a.v_col != 0 && a.dk <= 64 && a.dv <= 64 ? kLtBlock : kLtUnit;
  return s;
}

// Two CTAs per SM where half the shared memory holds a tile and a unit: while one waits for its scores or its
// probabilities, the other has products to run.  (64 columns need the registers of a whole SM.)
static int lt_per_sm(const LtShape& sh, long long items, int sms, int limit, int* units) {
  *units = sh.units((size_t)limit);
  if (sh.N < 64 && items > sms) {
    const int half = sh.units((size_t)(limit - 1024) / 2);  // each CTA costs another KB of the SM's 228
    if (half > sh.upt) {
      *units = half;
      return 2;
    }
  }
  return 1;
}

// Rows of one prompt that an item takes together: the number for which the rounds of items over the CTAs take the least
// time.  A tile's products cost the same for 16, 32 or 64 columns (A is read from shared memory at the same rate), its
// softmax does not: an item of 1000 prompt keys takes 27 us alone, 35 with 16 columns of several rows, 43 with 32
// and 68 with 64 (4 or 8 groups, heads of 128; latents of 256: 31, -, 39, 55; of 512: 53, -, 68, 90).  The keys of
// the rows themselves are no less work together: a short tile for two rows, or a whole one each.  1000 rows of one prompt of
// 1000, each by itself / together: 307 / 139 us (4 groups of 128), 588 / 237 (8 groups), 252 / 86 (4 groups of 64),
// 123 / 96 (latents of 256), 313 / 166 (of 512); 64 prompts with 4 rows each, latents of 512: 94 / 66; 150 with 3 rows, 300 keys, latents
// of 512, where it does not pay: 90 / 98.
// In tiles of one row: an item's start and end, a tile of its prompt, a tile of a row's own keys (half of one where they are 64 or fewer and two
// rows come in one), fitted to 14 jobs of 12 to 1200 rows for each of five shapes.  Two CTAs of an SM share its pipes.  Before the fit
// 1000 rows with 128 prompt keys and 200 of their own took 150 against 125 us (latents of 512), 162 against 136 (4 groups of 128).
static double lt_item_cost(const LatentArgs& a, const LtShape& sh, int rg, int per_sm) {
  const int prompt = (a.prompt_keys + kLtKeys - 1) / kLtKeys, tiles = a.own_keys > 0 ? (a.own_keys + kLtKeys - 1) / kLtKeys : 1;
  const bool pairs = a.own_keys <= kLtKeys / 2;
  if (a.v_col == 0) {
    if (rg == 1) return (per_sm == 2 ? 1.4 : 1.) * (0.5 + prompt + tiles);
    return sh.N == 64 ? 3.9 + 1.4 * prompt + rg * (pairs ? 0.57 : 1.3 * tiles) : 1.6 + 1.15 * prompt + rg * (pairs ? 0.75 : 1.2 * tiles);
  }
  if (rg == 1) return 2 + prompt + tiles;
  if (sh.N == 16) return 1.6 * prompt + rg * (pairs ? 1.1 : 2.3 * tiles);
  if (sh.N == 32) return (per_sm == 2 ? 1.4 : 1.) * (2.5 + 1.4 * prompt + rg * (pairs ? 0.67 : 1.15 * tiles));
  return 6.5 + 1.6 * prompt + rg * (pairs ? 1.05 : 1.4 * tiles);
}
static int lt_rows(const LatentArgs& a, int sms, int limit) {
  const int per = a.H / a.G;
  if (a.share < 2 || a.Tn != 1 || !a.kv.page_table || (per & (per - 1)) != 0) return 1;
  // Little to share: 1000 rows with 64 prompt keys and 400 of their own took 249 us with 4 rows together against 234 (4 groups of 128).
  if (!a.together && a.own_keys > kLtKeys / 2 && 2LL * a.prompt_keys < a.own_keys) return 1;
  const int cols = lt_cols(a);
  int best = 1;
  double least = 0.;
  for (int rg = 1; rg == 1 || rg * cols <= 64; rg *= 2) {
    if (rg > 1 && (rg > 2 * a.share || rg * cols < 16)) continue;
    const LtShape sh = lt_shape(a, rg);
    if (sh.units((size_t)limit) < sh.upt) continue;
    if (rg > 1 && cols < 16 && 2 * sh.N + sh.uv * (sh.N + 16 * rg) > 8 * sh.N) continue;  // TMEM
    if (rg == a.together) return rg;
    const long long items = (long long)(a.n_seq / a.share) * ((a.share + rg - 1) / rg) * a.G * a.n_splits;
    int units;
    const int per_sm = lt_per_sm(sh, items, sms, limit, &units);
    const long long ctas = (long long)per_sm * sms;
    const double t = (double)((items + ctas - 1) / ctas) * lt_item_cost(a, sh, rg, per_sm);
    if (rg == 1 || t < least) {
      least = t;
      best = rg;
    }
  }
  return a.together ? 1 : best;
}

template <int NB, int HS, bool SHARED, bool ROWS = false>
static int lt_launch(const CUtensorMap& mq, const CUtensorMap& mc, const LtParams& p, int grid, size_t smem, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(latent_tc_kernel<NB, HS, SHARED, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) {
    set_error("latent_attn: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    return DGPT_E_CUDA;
  }
  launch_few(p.n_rows <= kFewRows, latent_tc_kernel<NB, HS, SHARED, ROWS>, dim3(grid), dim3(kLtThreads), smem, st, mq, mc, p);
  return launch_status("latent_attn");
}

static void lt_device(int* sms, int* smem) {
  static int n_sm[64] = {}, n_smem[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (n_sm[dev] == 0) {
    cudaDeviceGetAttribute(&n_smem[dev], cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&n_sm[dev], cudaDevAttrMultiProcessorCount, dev);
  }
  *sms = n_sm[dev] > 0 ? n_sm[dev] : 1;
  *smem = n_smem[dev];
}

}  // namespace tc

bool latent_tc_supported(const LatentArgs& a, const dgpt_kv_layout& kv, int dtype) {
  if (dtype != DGPT_BF16 || a.dk > 512 || a.dv > 512) return false;
  const int pt = kv.page_tokens;
  if (kv.page_table && !((pt >= tc::kLtKeys && pt % tc::kLtKeys == 0) || (pt >= 8 && pt < tc::kLtKeys && tc::kLtKeys % pt == 0))) return false;
  if (kv.page_stride <= 0 || a.q_rs <= 0) return false;
  if (!tc::device_is_sm100() || tc::encode_fn() == nullptr) return false;
  int sms, smem;
  tc::lt_device(&sms, &smem);
  const tc::LtShape sh = tc::lt_shape(a, 1);
  return sh.units((size_t)smem) >= sh.upt;
}

int latent_tc_launch(const LatentArgs& a, const dgpt_kv_layout& kv, cudaStream_t st) {
  using namespace tc;
  int sms, limit;
  lt_device(&sms, &limit);
  const int rg = lt_rows(a, sms, limit);
  const LtShape sh = lt_shape(a, rg);
  const int N = sh.N;
  LtParams p;
  p.a = a;
  p.per = a.H / a.G;
  p.gpk = (p.per + N - 1) / N;
  p.n_rows = a.n_seq * a.Tn;
  p.n_groups = a.G * p.gpk;
  p.rg = rg;
  p.cols = lt_cols(a);
  p.cols_log2 = 0;
  while (1 << p.cols_log2 < p.cols) ++p.cols_log2;
  p.sets_per_prompt = rg > 1 ? (a.share + rg - 1) / rg : 1;
  p.n_sets = rg > 1 ? p.n_rows / a.share * p.sets_per_prompt : p.n_rows;
  p.n_items = p.n_sets * p.n_groups * a.n_splits;
  p.uk = sh.uk;
  p.uv = sh.uv;
  p.upt = sh.upt;
  p.unit_bytes = sh.unit_bytes;
  const int per_sm = lt_per_sm(sh, p.n_items, sms, limit, &p.n_units);
  const int pt = kv.page_tokens;
  p.box = kv.page_table && pt < kLtKeys ? pt : kLtKeys;
  p.align = kv.page_table ? p.box : 1;  // a dense run may be entered at any slot
  CUtensorMap mq, mc;
  {
    const cuuint64_t dims[3] = {(cuuint64_t)a.dk, (cuuint64_t)a.H, (cuuint64_t)p.n_rows};
    const cuuint64_t strides[2] = {(cuuint64_t)a.dk * 2, (cuuint64_t)a.q_rs * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)(N / rg), (cuuint32_t)rg};  // with several rows their heads make N
    if (!encode_3d(&mq, a.q, dims, strides, box)) return DGPT_E_CUDA;
  }
  {
    const cuuint64_t n_pages = kv.page_table ? (kv.n_pages > 0 ? (cuuint64_t)kv.n_pages : (cuuint64_t)1 << 24) : (cuuint64_t)a.n_seq;
    const cuuint64_t dims[3] = {(cuuint64_t)a.row_w, (cuuint64_t)pt, n_pages};
    const cuuint64_t strides[2] = {(cuuint64_t)a.row_w * 2, (cuuint64_t)kv.page_stride * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)p.box, 1};
    if (!encode_3d(&mc, kv.k_base, dims, strides, box)) return DGPT_E_CUDA;
  }
  const size_t smem = sh.bytes(p.n_units);
  const int grid = p.n_items < per_sm * sms ? p.n_items : per_sm * sms;
  if (rg > 1) {
#define DGPT_LT(NB, HS, SHARED) lt_launch<NB, HS, SHARED, true>(mq, mc, p, grid, smem, st)
    if (a.v_col == 0) return N == 32 ? DGPT_LT(2, 16, true) : DGPT_LT(4, 16, true);
    if (p.cols == 4) return N == 16 ? DGPT_LT(1, 4, false) : N == 32 ? DGPT_LT(2, 4, false) : DGPT_LT(4, 4, false);
    if (p.cols == 8) return N == 16 ? DGPT_LT(1, 8, false) : N == 32 ? DGPT_LT(2, 8, false) : DGPT_LT(4, 8, false);
    return N == 32 ? DGPT_LT(2, 16, false) : DGPT_LT(4, 16, false);
#undef DGPT_LT
  }
  if (a.v_col == 0) {
    if (N == 16) return lt_launch<1, 16, true>(mq, mc, p, grid, smem, st);
    if (N == 32) return lt_launch<2, 32, true>(mq, mc, p, grid, smem, st);
    return lt_launch<4, 64, true>(mq, mc, p, grid, smem, st);
  }
  if (p.per <= 4) return lt_launch<1, 4, false>(mq, mc, p, grid, smem, st);
  if (p.per <= 8) return lt_launch<1, 8, false>(mq, mc, p, grid, smem, st);
  if (N == 16) return lt_launch<1, 16, false>(mq, mc, p, grid, smem, st);
  if (N == 32) return lt_launch<2, 32, false>(mq, mc, p, grid, smem, st);
  return lt_launch<4, 64, false>(mq, mc, p, grid, smem, st);
}

}  // namespace dgpt
