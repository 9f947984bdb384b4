// Whole forwards of a small fp32 GPT (n_embd 32, 64 or 128) in one launch, and whole decode loops: what such a model does per token is a
// hundred thousand multiply-adds, so that a step made of one launch per product is nothing but launches (24 of them, 85 us a step of
// 100 futures; the rows themselves need no one's result but their own).
//
//   decode    a CTA owns M rows from the first step to the last: embedding, layers, head, draw, and again.  No grid-wide wait; a row's
//             K/V goes to its pages and is read back from there by the same CTA.
//   chunk     up to 16 M tokens of one sequence (a prompt, or a portion of one): a cluster, each CTA M tokens.  After a layer's K/V has
//             been appended the cluster waits once, and every token then reads the keys before it.
//
// What bounds it: the latency of some nine dependent phases a layer, 700 to 2000 clocks each.  The weights (11 C^2 a layer) pass through
// every CTA once per forward, 420 KB for 2 layers of 64 with a head of 256; a warp of its own streams them from L2 through a ring in
// shared memory (cp.async.bulk), so that neither their latency nor the load pipe they would fill stands in the way of the phases.  (Read
// straight into registers, 8 words a thread ahead: 22 us a step, the loads holding up the shared-memory reads behind them.)  Eight warps
// and not sixteen: half the instructions that every warp repeats, and registers enough that nothing is spilled.
// Measured: 100 futures of 2 layers of 64 (fp32, 89 + 48 keys) 85 us a step as 24 launches, 12.8 here; 1000 of them 85 -> 60.
// M = 1 up to as many rows as SMs, else 2, 4 or 8: the weights are then read once for M rows.
#include "small_gpt.cuh"

namespace dgpt {

int small_gpt_64(const SmallGpt& p, int M, int grid, cudaStream_t st) { return small_gpt_pick<64>(p, M, grid, st); }

static int small_gpt_dispatch(const SmallGpt& p, int C, int M, int grid, cudaStream_t st) {
  return C == 32 ? small_gpt_32(p, M, grid, st) : C == 64 ? small_gpt_64(p, M, grid, st) : small_gpt_128(p, M, grid, st);
}

}  // namespace dgpt

using namespace dgpt;

extern "C" int dgpt_small_gpt_supported(int32_t C, int32_t H, int32_t L, int32_t V, int32_t max_keys) {
  if (!(C == 32 || C == 64 || C == 128) || H <= 0 || C % H != 0 || L < 1 || L > kSgMaxLayers || V < 4 || V % 4 != 0 || V > 4096) return 0;
  const int D = C / H;
  if (!(D == 8 || D == 16 || D == 32) || max_keys < 1 || max_keys > (1 << 14)) return 0;
  return small_gpt_smem(C, 1, L, H, V, true, max_keys, false) <= kSgRest && small_gpt_smem(C, 8, L, H, V, false, max_keys, true) <= kSgRest;
}

extern "C" int dgpt_small_gpt(const dgpt_small_gpt_model* model, const dgpt_kv_layout* kv, int64_t kv_layer_stride, const int32_t* ids,
                              const int32_t* pos0, const int32_t* slot0, const int32_t* step_ptr, const int32_t* len0,
                              const int32_t* start1, const int32_t* len1, int32_t n_seq, int32_t T, int32_t max_keys, int32_t last_only, float* logits,
                              float logit_cap, int32_t n_steps, const dgpt_small_gpt_draw* draw, int32_t* status, void* stream) {
  DGPT_REQUIRE(model && model->emb && model->weights && model->cs_table && ids && pos0 && slot0 && logits && status,
               "small_gpt: NULL pointer");
  const dgpt_small_gpt_model& m = *model;
  if (!dgpt_small_gpt_supported(m.C, m.H, m.L, m.V, max_keys)) {
    set_error("small_gpt: %d layers of %d with %d heads, a vocabulary of %d and %d keys are not built", m.L, m.C, m.H, m.V, max_keys);
    return DGPT_E_UNSUPPORTED;
  }
  DGPT_REQUIRE(n_seq >= 0 && T >= 0 && m.layers_per_block >= 1 && m.table_len > 0, "small_gpt: bad sizes");
  DGPT_REQUIRE(T > 0 || (n_steps >= 1 && len1), "small_gpt: a decode step needs its keys' number");
  DGPT_REQUIRE(T == 0 || (n_steps == 1 && !draw), "small_gpt: tokens of a sequence are one forward without a draw");
  DGPT_REQUIRE(n_steps == 1 || draw, "small_gpt: several steps need a draw");
  DGPT_REQUIRE(!draw || (draw->out_tokens && draw->history && draw->traj_ids), "small_gpt: NULL pointer in the draw");
  DGPT_REQUIRE(!draw || (draw->temperature >= 0.f && draw->cap >= 0.f), "small_gpt: temperature and cap must be non-negative");
  if (((reinterpret_cast<uintptr_t>(m.weights) | reinterpret_cast<uintptr_t>(kv ? kv->k_base : nullptr)) & 15) != 0) {
    set_error("small_gpt: weights must be 16-byte aligned");
    return DGPT_E_UNSUPPORTED;
  }
  int rc = validate_kv(kv, m.C / m.H);
  if (rc != DGPT_OK) return rc;
  DGPT_REQUIRE(kv_layer_stride % 4 == 0, "small_gpt: the layers' stride must be a multiple of 4");
  if (n_seq == 0) return DGPT_OK;
  const long long span = (kv->page_table ? kv->n_pages : n_seq) * (long long)kv->page_stride;
  if ((kv->page_table && kv->n_pages <= 0) || span / 4 >= (long long)kNoKey) {
    set_error("small_gpt: the cache's size must be stated and below 64 GB a layer");
    return DGPT_E_UNSUPPORTED;
  }
  SmallGpt p = {};
  p.max_keys = max_keys;
  p.emb = m.emb;
  p.w = m.weights;
  p.n_w = (long long)m.L * 11 * m.C * m.C + (long long)((m.V + 255) / 256) * 256 * m.C;
  p.cs = m.cs_table;
  p.kv = make_view(kv);
  p.layer_stride = kv_layer_stride;
  p.ids = ids;
  p.pos0 = pos0;
  p.slot0 = slot0;
  p.step = step_ptr;
  p.len0 = len0;
  p.start1 = start1;
  p.len1 = T > 0 ? nullptr : len1;
  p.logits = logits;
  p.status = status;
  p.L = m.L;
  p.H = m.H;
  p.V = m.V;
  p.layers_per_block = m.layers_per_block;
  p.table_len = m.table_len;
  p.R = n_seq;
  p.last_only = T > 0 ? last_only : 0;
  p.n_steps = n_steps;
  p.alpha = m.swiglu_alpha;
  p.limit = m.swiglu_limit;
  p.logit_cap = logit_cap;
  p.cluster = 1;
  if (draw) {
    p.cap = draw->cap;
    p.temperature = draw->temperature;
    p.top_p = draw->top_p;
    p.seed_lo = (uint32_t)draw->seed;
    p.seed_hi = (uint32_t)(draw->seed >> 32);
    while ((32 << p.log2c) < m.V) ++p.log2c;
    p.force_rows = draw->force_group_rows > 0 ? draw->force_group_rows : 1;
    p.traj = reinterpret_cast<const long long*>(draw->traj_ids);
    p.force = draw->force_schedule;
    p.force_stride = draw->force_group_stride;
    p.hist_stride = draw->history_stride;
    p.out_tok = draw->out_tokens;
    p.hist = draw->history;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  if (T == 0) {
    int M = 1;
    while (M < 8 && M * sms < n_seq && small_gpt_smem(m.C, 2 * M, m.L, m.H, m.V, draw != nullptr, max_keys, false) <= kSgRest) M *= 2;
    return small_gpt_dispatch(p, m.C, M, (n_seq + M - 1) / M, st);
  }
  p.T_all = T;
  for (int t = 0; t < T;) {  // up to 16 CTAs of up to 8 tokens each at a time
    const int n = T - t < 128 ? T - t : 128;
    int M = 1;
    while (M < 8 && (M * 16 < n || (long long)n_seq * ((n + M - 1) / M) > sms)) M *= 2;
    p.T = n;
    p.t_base = t;
    p.cluster = (n + M - 1) / M;
    rc = small_gpt_dispatch(p, m.C, M, n_seq * p.cluster, st);
    if (rc != DGPT_OK) return rc;
    t += n;
  }
  return DGPT_OK;
}
