// Library identity, workspace carving and the whole-layer entry points.
#include "common.cuh"
#include "shared_role.cuh"

namespace b200moe {

static size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct Workspace {
  float* w;               // [T][4]
  int32_t* ids;           // [T][4]
  int32_t* sorted_ids;    // [R]
  float* sorted_w;        // [R]
  int32_t* block_expert;  // [R/bm]
  int32_t* num_valid;     // [2]
  int32_t* scratch;       // permute chunk counts
  uint8_t* xq_sorted;     // [R][3072]
  uint8_t* sfx;           // [R/bm][48][512]
  uint8_t* hq;            // [R][384]
  uint8_t* sfh;           // [R/bm][6][512]
  int32_t* done;          // [R/bm] GEMM1 tiles finished per row block, then [kSharedDone]: the shared expert's
  float* partials;        // [S][T][E] split-K logit partials; only with the router inside the call
  uint8_t* q4;            // [T][3072] row-major MXFP4 codes of x or rebuilt from a compact input; not where up to 32 tokens with
  uint8_t* s4;            // [T][192] their scales                        logits are quantised on the way into sorted order
  // only with the shared expert:
  SharedWorkspace sh;
  bool sum_in_gemm2;          // nobody takes the shared rows: the shared expert's second GEMM sums the slots (shared_pair.cu, MODE 3)
  // results the caller does not take:
  __nv_bfloat16* shared_out;  // [T][6144]; not with sum_in_gemm2
  __nv_bfloat16* slots;       // [T][4][6144]
  size_t bytes;
  int bm;
  int64_t rows;
};

int dispatch_rows_done(const uint8_t* codes, const uint8_t* scales, const int32_t* sorted_ids, const int32_t* num_valid,
                       int64_t tokens, int bm, int by_pair, int64_t max_rows, uint8_t* xq_sorted, uint8_t* sfx,
                       int32_t* done, int n_done, void* stream);
int prep_small(const float* partials, int64_t stride_t, int64_t stride_s, int splits, const float* bias, int64_t tokens,
               int num_experts, int mode, float scale, int bm, float* out_w, int32_t* out_ids, int32_t* sorted_ids,
               float* sorted_w, int32_t* block_expert, int32_t* num_valid, const void* x_bf16, const uint8_t* q4,
               const uint8_t* s4, int64_t max_rows, uint8_t* xq_sorted, uint8_t* sfx, int32_t* done, int n_done,
               void* stream);
int quant_rows_both(const void* x_bf16, int64_t tokens, uint8_t* codes, uint8_t* scales, uint8_t* codes8, uint8_t* scales8,
                    uint8_t* atoms8, int bm8, void* stream);
int route_quant(const float* logits, const float* bias, int64_t tokens, int num_experts, int mode, float scale, const void* x_bf16,
                float* out_w, int32_t* out_ids, uint8_t* codes4, uint8_t* scales4, uint8_t* codes8, uint8_t* atoms8, int bm8,
                void* stream);
int router_tc_quant(const void* x_bf16, const void* gate_split_bf16, int64_t tokens, int num_experts, int splits, float* partials,
                    uint8_t* codes4, uint8_t* scales4, uint8_t* codes8, uint8_t* scales8, uint8_t* atoms8, int bm8, int32_t* status,
                    void* stream);
int router_gemm_quant(const void* x_bf16, const float* gate, int64_t tokens, int num_experts, int splits, float* partials,
                      uint8_t* codes4, uint8_t* scales4, uint8_t* codes8, uint8_t* scales8, uint8_t* atoms8, int bm8,
                      void* stream);
int gemm12_beside(const uint8_t* w13t, const uint8_t* w2t, int num_experts, const uint8_t* xq_sorted, const uint8_t* sfx,
                  const int32_t* block_expert, const int32_t* num_valid, const int32_t* sorted_ids, const float* sorted_w,
                  int64_t max_rows, int bm, int64_t tokens, uint8_t* hq, uint8_t* sfh, int32_t* done, void* slots_bf16,
                  int32_t* status, const SharedPlan* sp, void* stream);
int gemm1_beside(const uint8_t* w13t, int num_experts, const uint8_t* xq_sorted, const uint8_t* sfx,
                 const int32_t* block_expert, const int32_t* num_valid, int64_t max_rows, int bm, uint8_t* hq, uint8_t* sfh,
                 const uint8_t* prefetch_w2t, int32_t* status, const SharedPlan* sp, void* stream);
int sidecar_unpack_atoms(const uint8_t* mask, const uint8_t* s4, const uint8_t* q8, const uint8_t* s8, int64_t tokens, uint8_t* q4,
                         uint8_t* atoms, int bm, void* stream);
int shared_gemm1(const uint8_t* w13t, const uint8_t* codes8, int64_t code_rows, const SharedWorkspace& ws, int64_t tokens,
                 int32_t* status, void* stream);
bool shared_sums_slots(const SharedWorkspace& ws);
int shared_gemm2(const uint8_t* w2t, const SharedWorkspace& ws, const void* slots_bf16, void* out_bf16, int64_t tokens,
                 int32_t* status, void* stream);
int set_wait_limit_routed(unsigned long long ns);
int set_wait_limit_shared(unsigned long long ns);
int set_wait_limit_shared_pair(unsigned long long ns);
int set_wait_limit_pair(unsigned long long ns);
int set_wait_limit_router(unsigned long long ns);
int set_wait_limit_ep_sync(unsigned long long ns);

constexpr int64_t kSmallTokens = 32;  // up to here routing, sort and gather are one launch

static Workspace carve(uint8_t* base, int64_t tokens, int num_experts, int flags) {
  Workspace ws{};
  ws.bm = b200moe_block_rows(tokens);
  ws.rows = b200moe_max_sorted_rows(tokens, ws.bm, num_experts);
  const size_t blocks = static_cast<size_t>(ws.rows / ws.bm);
  size_t off = 0;
  auto take = [&](size_t n) {
    uint8_t* p = base ? base + off : nullptr;
    off = align_up(off + n, 1024);
    return p;
  };
  ws.w = reinterpret_cast<float*>(take(tokens * kTopK * 4));
  ws.ids = reinterpret_cast<int32_t*>(take(tokens * kTopK * 4));
  ws.sorted_ids = reinterpret_cast<int32_t*>(take(ws.rows * 4));
  ws.sorted_w = reinterpret_cast<float*>(take(ws.rows * 4));
  ws.block_expert = reinterpret_cast<int32_t*>(take(blocks * 4));
  ws.num_valid = reinterpret_cast<int32_t*>(take(16));
  ws.scratch = reinterpret_cast<int32_t*>(take(b200moe_permute_scratch_bytes(tokens, num_experts) + 16));
  if (ws.bm < 128) {  // at block height 128 GEMM1 gathers its rows itself
    ws.xq_sorted = take(ws.rows * (kH / 2));
    ws.sfx = take(blocks * (kH / 128) * kAtomBytes);
  }
  ws.hq = take(ws.rows * (kI / 2));
  ws.sfh = take(blocks * (kI / 128) * kAtomBytes);
  ws.done = reinterpret_cast<int32_t*>(take((blocks + kSharedDone) * 4));
  if (flags & B200MOE_LAYER_ROUTER)
    ws.partials = reinterpret_cast<float*>(take(static_cast<size_t>(b200moe_router_splits(tokens)) * tokens * num_experts * 4));
  if ((flags & (B200MOE_LAYER_ROUTER | B200MOE_LAYER_COMPACT)) || tokens > kSmallTokens) {
    ws.q4 = take(tokens * (kH / 2));
    ws.s4 = take(tokens * (kH / 32));
  }
  if (flags & B200MOE_LAYER_SHARED) {
    ws.sh = carve_shared(nullptr, tokens);
    uint8_t* p = take(ws.sh.bytes);
    if (p) ws.sh = carve_shared(p, tokens);
    if (flags & B200MOE_LAYER_OWN_SHARED_OUT) {
      ws.sum_in_gemm2 = ws.bm == 128 && shared_sums_slots(ws.sh);
      if (!ws.sum_in_gemm2) ws.shared_out = reinterpret_cast<__nv_bfloat16*>(take(tokens * kH * 2));
    }
  }
  if (flags & B200MOE_LAYER_OWN_SLOTS) ws.slots = reinterpret_cast<__nv_bfloat16*>(take(tokens * kTopK * kH * 2));
  ws.bytes = off;
  return ws;
}

}  // namespace b200moe

extern "C" int b200moe_version(void) { return 1; }
extern "C" const char* b200moe_arch(void) { return "sm_100a"; }

extern "C" size_t b200moe_layer_workspace_bytes(int64_t tokens, int num_experts, int flags) {
  if (tokens < 1 || tokens > B200MOE_MAX_TOKENS || num_experts < 1 || num_experts > b200moe::kMaxE) return 0;
  return b200moe::carve(nullptr, tokens, num_experts, flags).bytes;
}

extern "C" size_t b200moe_workspace_bytes(int64_t tokens, int num_experts) {
  return b200moe_layer_workspace_bytes(tokens, num_experts, 0);
}

extern "C" size_t b200moe_workspace_bytes_x(int64_t tokens, int num_experts) {
  return b200moe_layer_workspace_bytes(tokens, num_experts, B200MOE_LAYER_ROUTER);
}

extern "C" int b200moe_set_wait_limit_ns(uint64_t ns) {
  if (ns == 0) return B200MOE_E_ARG;
  int r = b200moe::set_wait_limit_routed(ns);
  if (!r) r = b200moe::set_wait_limit_shared(ns);
  if (!r) r = b200moe::set_wait_limit_shared_pair(ns);
  if (!r) r = b200moe::set_wait_limit_pair(ns);
  if (!r) r = b200moe::set_wait_limit_router(ns);
  if (!r) r = b200moe::set_wait_limit_ep_sync(ns);
  return r;
}

namespace b200moe {
// Both grouped GEMMs in one persistent launch: up to 32 tokens, and with I = 1536 wherever the row blocks have 16 rows (up to 480).
// Measured, whole layer, two launches / one, us: I = 1536 287 / 255 at 64 tokens, 330 / 294 at 128, 355 / 318 at 400 (router and
// shared expert inside: 318 / 298, 342 / 321, 385 / 367): 24 W13 tiles of an expert leave more of an unfinished last round, and
// GEMM2 fills it. I = 768: 114 / 111 at 33, 141 / 139 at 64, 171 / 171 at 128, 179 / 184 at 400 (181 / 187 at 128 with both inside).
static bool one_launch(int64_t tokens, int bm) { return tokens <= kSmallTokens || (kI == 1536 && bm == 16); }

// One call of the layer, in any of its forms.
struct LayerCall {
  const b200moe_weights* w;
  const b200moe_shared_weights* shared;  // null: routed experts only
  const void* x;                         // bf16 rows, or (null) a prepared input:
  const b200moe_prepared* prep;
  const float* logits;                   // with x: plain logits, null: the router runs inside the call
  int64_t tokens;
  void* workspace;
  size_t workspace_bytes;
  void *slots, *shared_out, *out;
  int32_t* status;
  void* stream;
  void* side;  // may be null: another stream of the device, for the shared expert's GEMMs above 512 tokens (the first only, where
               // the second sums the slots behind GEMM2)
};

// The side stream's part of a call: starts behind what the main stream holds at fork() and is joined by join(), at the latest when
// the call returns, error returns included (a capture must not end with an unjoined stream, and the caller frees the workspace in
// main-stream order). Both events live for the call only, so calls from several threads and streams share nothing.
class SideStream {
 public:
  SideStream(void* main, void* side) : main_(static_cast<cudaStream_t>(main)), side_(static_cast<cudaStream_t>(side)) {}
  ~SideStream() {
    (void)join();
    if (begin_) cudaEventDestroy(begin_);
    if (end_) cudaEventDestroy(end_);
  }
  int fork() {
    cudaError_t e = cudaEventCreateWithFlags(&begin_, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&end_, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventRecord(begin_, main_);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(side_, begin_, 0);
    forked_ = e == cudaSuccess;
    return static_cast<int>(e);
  }
  int join() {
    if (!forked_) return 0;
    forked_ = false;
    cudaError_t e = cudaEventRecord(end_, side_);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(main_, end_, 0);
    return static_cast<int>(e);
  }

 private:
  cudaStream_t main_, side_;
  cudaEvent_t begin_ = nullptr, end_ = nullptr;
  bool forked_ = false;
};

// Logits given and a shared expert on the side stream: where the routing stays a launch of its own behind the quantisers. The
// side stream starts when x is quantised, and its first GEMM takes every SM, as GEMM1 does: whichever is there first, the other
// waits. With a routing launch in front of the sort the shared GEMM is first and hides the routing and the sort; without
// (route_quant) the early launches of the chain put GEMM1 first, and the shared GEMMs run against its tail and GEMM2's. That is
// the better order again where GEMM2 and the shared rows are stored side by side, from 18 blocks of 128 tokens on, and where the
// slots are summed from 44 on. Measured, the layer with logits, one launch / two, us: I = 768 reduced 231 / 236 at 1152 tokens,
// 233 / 235 at 1153, 246 / 236 at 1183, 248 / 243 at 1408, 260 / 252 at 1800, 274 / 265 at 2176, (the exception:) 269 / 277 at
// 2200, 278 / 267 at 2304, 279 / 263 at 2560, 292 / 288 at 3072, 437 / 427 at 5120, 461 / 456 at 5632, 477 / 487 at 5900, 826 /
// 855 at 12288, 1075 / 1095 at 16384; slots handed out 237 / 240 at 1152, 252 / 242 at 1183, 273 / 261 at 1800, 303 / 286 at
// 2240, 299 / 278 at 2280, 304 / 302 at 2299, 321 / 326 at 3072, 383 / 403 at 4096, 1174 / 1242 at 16384. I = 1536 reduced 414 /
// 400 at 1280, 453 / 437 at 2176, 486 / 476 at 3072; slots handed out 435 / 410 at 1280, 500 / 483 at 2240, 494 / 501 at 2299,
// 574 / 594 at 3328.
constexpr int64_t kRouteBehindFrom = 9 * 128 + 1, kRouteBehindToStored = 18 * 128, kRouteBehindToSummed = 44 * 128;
static bool routes_behind_quant(const LayerCall& c, const Workspace& ws) {
  return c.x && c.logits && c.shared && c.side && c.tokens >= kRouteBehindFrom &&
         c.tokens <= (ws.sum_in_gemm2 ? kRouteBehindToSummed : kRouteBehindToStored);
}

static int run_layer(const LayerCall& c) {
  const b200moe_weights* w = c.w;
  if (!w || !c.workspace || !c.status || (!c.x == !c.prep) || (!c.slots && !c.out)) return B200MOE_E_ARG;
  if (c.tokens < 1 || c.tokens > B200MOE_MAX_TOKENS) return B200MOE_E_ARG;
  const bool shared = c.shared != nullptr, router = c.x && !c.logits, compact = c.prep && c.prep->mask4;
  if (router && !w->gate) return B200MOE_E_ARG;
  if (shared && (!c.shared->w13t || !c.shared->w2t || (!c.shared_out && !c.out))) return B200MOE_E_ARG;
  if (shared && c.shared->intermediate != 0 && c.shared->intermediate != kI) return B200MOE_E_ARG;
  if (c.prep && (!c.prep->scales4 || !c.prep->topk_weights || !c.prep->topk_ids || (!c.prep->codes4 && !compact) ||
                 ((shared || compact) && (!c.prep->codes8 || !c.prep->scales8))))
    return B200MOE_E_ARG;
  if (reinterpret_cast<uintptr_t>(c.workspace) & 255) return B200MOE_E_ALIGN;
  // (with the router inside, its GEMM takes any row address below 128 tokens and says what it needs above)
  if (c.x && c.logits && (reinterpret_cast<uintptr_t>(c.x) & 15)) return B200MOE_E_ALIGN;
  if (shared && ((reinterpret_cast<uintptr_t>(c.shared->w13t) | reinterpret_cast<uintptr_t>(c.shared->w2t) |
                  reinterpret_cast<uintptr_t>(c.shared_out)) & 15))
    return B200MOE_E_ALIGN;
  // (the rebuild of a compact input checks its own operands: 8 bytes for the FP8 codes)
  if (c.prep && ((reinterpret_cast<uintptr_t>(c.prep->codes4) | (shared ? reinterpret_cast<uintptr_t>(c.prep->codes8) : 0)) & 15))
    return B200MOE_E_ALIGN;
  // the last launch reads the slots and writes `out` 16 bytes at a time, whichever kernel it is (the slot reduce or the shared expert's
  // second GEMM); GEMM2 writes the slots in pieces of 16 bytes from blocks of 128 rows, of 8 bytes from smaller ones
  const uintptr_t slot_bytes = c.out || b200moe_block_rows(c.tokens) == 128 ? 16 : 8;
  if ((reinterpret_cast<uintptr_t>(c.out) & 15) || (reinterpret_cast<uintptr_t>(c.slots) & (slot_bytes - 1))) return B200MOE_E_ALIGN;
  const int ne = w->num_experts;
  const int64_t tokens = c.tokens;
  void* st = c.stream;
  int flags = 0;
  if (router) flags |= B200MOE_LAYER_ROUTER;
  if (compact) flags |= B200MOE_LAYER_COMPACT;
  if (shared) flags |= B200MOE_LAYER_SHARED;
  if (shared && !c.shared_out) flags |= B200MOE_LAYER_OWN_SHARED_OUT;
  if (!c.slots) flags |= B200MOE_LAYER_OWN_SLOTS;
  const Workspace ws = carve(static_cast<uint8_t*>(c.workspace), tokens, ne, flags);
  if (c.workspace_bytes < ws.bytes) return B200MOE_E_ARG;
  void* slots = c.slots ? c.slots : ws.slots;
  void* shared_out = c.shared_out ? c.shared_out : ws.shared_out;
  const int blocks = static_cast<int>(ws.rows / ws.bm), n_done = blocks + (shared ? kSharedDone : 0);
  const int splits = router ? b200moe_router_splits(tokens) : 1;
  const float* partials = router ? ws.partials : c.logits;
  const int64_t stride_s = router ? tokens * ne : 0;
  const uint8_t *q4 = c.prep ? c.prep->codes4 : ws.q4, *s4 = c.prep ? c.prep->scales4 : ws.s4;
  const uint8_t* codes8 = c.prep ? c.prep->codes8 : ws.sh.x8;
  bool have_q4 = true, routed = c.prep != nullptr;  // the tokens are quantised / routed
  int r = 0;
  SideStream side(c.stream, c.side);
  // the operands: quantised rows and, with the router inside, the logits' split-K partials
  if (c.prep) {
    if (compact) {
      r = sidecar_unpack_atoms(c.prep->mask4, s4, codes8, c.prep->scales8, tokens, ws.q4, shared ? ws.sh.sfx8 : nullptr, ws.sh.bm, st);
      if (r) return r;
      q4 = ws.q4;
    } else if (shared && (r = b200moe_scales_to_atoms(c.prep->scales8, tokens, kH / 32, ws.sh.bm, ws.sh.sfx8, st))) return r;
  } else if (router && (tokens < 128 || !w->gate_split)) {  // one pass over x
    r = router_gemm_quant(c.x, w->gate, tokens, ne, splits, ws.partials, ws.q4, ws.s4, shared ? ws.sh.x8 : nullptr, nullptr,
                          shared ? ws.sh.sfx8 : nullptr, ws.sh.bm, st);
    if (r) return r;
  } else if (router) {  // the same from 128 tokens on, the logits on the tensor cores
    r = router_tc_quant(c.x, w->gate_split, tokens, ne, splits, ws.partials, ws.q4, ws.s4, shared ? ws.sh.x8 : nullptr, nullptr,
                        shared ? ws.sh.sfx8 : nullptr, ws.sh.bm, c.status, st);
    if (r) return r;
  } else if (routes_behind_quant(c, ws)) {
    r = quant_rows_both(c.x, tokens, ws.q4, ws.s4, ws.sh.x8, nullptr, ws.sh.sfx8, ws.sh.bm, st);
    if (r) return r;
  } else if (tokens > kSmallTokens) {  // logits given: the routing beside the quantisers
    routed = true;
    r = route_quant(c.logits, w->bias, tokens, ne, w->route_mode, w->route_scale, c.x, ws.w, ws.ids, ws.q4, ws.s4,
                    shared ? ws.sh.x8 : nullptr, shared ? ws.sh.sfx8 : nullptr, ws.sh.bm, st);
    if (r) return r;
  } else {  // a few tokens: the routed rows are quantised by the launch that routes and sorts
    have_q4 = false;
    if (shared && (r = b200moe_shared_quant(c.x, tokens, ws.sh.bm, ws.sh.x8, ws.sh.sfx8, st))) return r;
  }
  SharedPlan plan{};
  const SharedPlan* sp = nullptr;
  if (shared) {
    if (ws.bm < 128) {  // decode sizes: a role of the launch that streams the routed experts' W13
      if ((r = shared_plan(&plan, c.shared->w13t, c.shared->w2t, codes8, tokens, ws.sh, shared_out, tokens, ws.done + blocks,
                           one_launch(tokens, ws.bm))))
        return r;
      sp = &plan;
    } else {  // beside the routing and the sort, whose few short launches leave the SMs to it
      if (c.side && (r = side.fork())) return r;
      void* sst = c.side ? c.side : st;
      r = shared_gemm1(c.shared->w13t, codes8, tokens, ws.sh, tokens, c.status, sst);
      if (!r && !ws.sum_in_gemm2) r = shared_gemm2(c.shared->w2t, ws.sh, nullptr, shared_out, tokens, c.status, sst);
      if (r) return r;
    }
  }

  // routing, sort, and at decode sizes the gather into sorted order
  if (!c.prep && tokens <= kSmallTokens && ne >= 4) {  // one launch
    r = prep_small(partials, ne, stride_s, splits, w->bias, tokens, ne, w->route_mode, w->route_scale, ws.bm, ws.w, ws.ids,
                   ws.sorted_ids, ws.sorted_w, ws.block_expert, ws.num_valid, have_q4 ? nullptr : c.x,
                   have_q4 ? q4 : nullptr, have_q4 ? s4 : nullptr, ws.rows, ws.xq_sorted, ws.sfx, ws.done, n_done, st);
    if (r) return r;
  } else {
    if (routed)
      r = b200moe_permute(c.prep ? c.prep->topk_ids : ws.ids, c.prep ? c.prep->topk_weights : ws.w, tokens, ne, ws.bm, ws.sorted_ids,
                          ws.sorted_w, ws.block_expert, ws.num_valid, ws.scratch, st);
    else
      r = b200moe_route_sort_partials(partials, ne, stride_s, splits, w->bias, tokens, ne, w->route_mode, w->route_scale, ws.bm,
                                      ws.w, ws.ids, ws.sorted_ids, ws.sorted_w, ws.block_expert, ws.num_valid, ws.scratch, st);
    if (r) return r;
    if (ws.bm < 128) {
      r = dispatch_rows_done(q4, s4, ws.sorted_ids, ws.num_valid, tokens, ws.bm, 0, ws.rows, ws.xq_sorted, ws.sfx, ws.done, n_done, st);
      if (r) return r;
    }
  }

  // the routed experts
  if (one_launch(tokens, ws.bm)) {
    r = gemm12_beside(w->w13t, w->w2t, ne, ws.xq_sorted, ws.sfx, ws.block_expert, ws.num_valid, ws.sorted_ids, ws.sorted_w,
                      ws.rows, ws.bm, tokens, ws.hq, ws.sfh, ws.done, slots, c.status, sp, st);
    if (r) return r;
  } else {
    if (ws.bm < 128)
      r = gemm1_beside(w->w13t, ne, ws.xq_sorted, ws.sfx, ws.block_expert, ws.num_valid, ws.rows, ws.bm, ws.hq, ws.sfh, w->w2t,
                       c.status, sp, st);
    else  // GEMM1 gathers its token rows from the row-major quantised tokens by the sorted list
      r = b200moe_gemm1_swiglu_quant_gather(w->w13t, ne, q4, s4, tokens, 0, ws.sorted_ids, ws.block_expert, ws.num_valid,
                                            ws.rows, ws.hq, ws.sfh, c.status, st);
    if (r) return r;
    if ((r = b200moe_gemm2_weighted(w->w2t, ne, ws.hq, ws.sfh, ws.block_expert, ws.num_valid, ws.sorted_ids, ws.sorted_w,
                                    ws.rows, ws.bm, tokens, slots, c.status, st)))
      return r;
  }
  if ((r = side.join())) return r;
  if (ws.sum_in_gemm2) return shared_gemm2(c.shared->w2t, ws.sh, slots, c.out, tokens, c.status, st);
  if (c.out && (r = b200moe_reduce_slots(slots, shared ? shared_out : nullptr, tokens, c.out, st))) return r;
  return 0;
}
}  // namespace b200moe

extern "C" int b200moe_layer(const b200moe_weights* w, const b200moe_shared_weights* shared, const void* x_bf16,
                             const float* logits, int64_t tokens, void* workspace, size_t workspace_bytes, void* slots_bf16,
                             void* shared_out_bf16, void* out_bf16, int32_t* status, void* stream,
                             void* side_stream) {
  return b200moe::run_layer({w, shared, x_bf16, nullptr, logits, tokens, workspace, workspace_bytes, slots_bf16,
                             shared_out_bf16, out_bf16, status, stream, side_stream});
}

extern "C" int b200moe_layer_prepared(const b200moe_weights* w, const b200moe_shared_weights* shared,
                                      const b200moe_prepared* input, int64_t tokens, void* workspace, size_t workspace_bytes,
                                      void* slots_bf16, void* shared_out_bf16, void* out_bf16, int32_t* status,
                                      void* stream, void* side_stream) {
  return b200moe::run_layer({w, shared, nullptr, input, nullptr, tokens, workspace, workspace_bytes, slots_bf16,
                             shared_out_bf16, out_bf16, status, stream, side_stream});
}

extern "C" int b200moe_prepare(const b200moe_weights* w, const void* x_bf16, int64_t tokens, float* partials, uint8_t* codes4,
                               uint8_t* scales4, float* topk_weights, int32_t* topk_ids, uint8_t* codes8, uint8_t* scales8,
                               int32_t* status, void* stream) {
  using namespace b200moe;
  if (!w || !w->gate || !x_bf16 || !partials || !codes4 || !scales4 || !topk_weights || !topk_ids || !status)
    return B200MOE_E_ARG;
  if (tokens < 1 || tokens > B200MOE_MAX_TOKENS || (codes8 != nullptr) != (scales8 != nullptr)) return B200MOE_E_ARG;
  const int ne = w->num_experts, splits = b200moe_router_splits(tokens);
  int r;
  if (tokens < 128 || !w->gate_split) {
    r = router_gemm_quant(x_bf16, w->gate, tokens, ne, splits, partials, codes4, scales4, codes8, scales8, nullptr, 16, stream);
  } else {
    r = router_tc_quant(x_bf16, w->gate_split, tokens, ne, splits, partials, codes4, scales4, codes8, scales8, nullptr, 16, status,
                        stream);
  }
  if (r) return r;
  return b200moe_route_topk(partials, ne, tokens * ne, splits, w->bias, tokens, ne, w->route_mode, w->route_scale, topk_weights,
                            topk_ids, stream);
}

extern "C" int b200moe_forward_x(const b200moe_weights* w, const void* x_bf16, int64_t tokens, void* workspace,
                                 size_t workspace_bytes, void* slots_bf16, void* out_bf16, int32_t* status,
                                 void* stream) {
  if (!slots_bf16) return B200MOE_E_ARG;
  return b200moe_layer(w, nullptr, x_bf16, nullptr, tokens, workspace, workspace_bytes, slots_bf16, nullptr, out_bf16, status,
                       stream, nullptr);
}

extern "C" int b200moe_forward(const b200moe_weights* w, const void* x_bf16, const float* logits, int64_t tokens,
                               void* workspace, size_t workspace_bytes, void* slots_bf16, void* out_bf16,
                               int32_t* status, void* stream) {
  if (!slots_bf16 || !logits) return B200MOE_E_ARG;
  return b200moe_layer(w, nullptr, x_bf16, logits, tokens, workspace, workspace_bytes, slots_bf16, nullptr, out_bf16, status,
                       stream, nullptr);
}

extern "C" int b200moe_forward_host(const b200moe_weights* w, const void* host_x_bf16, const float* host_logits,
                                    int64_t tokens, void* dev_x, float* dev_logits, void* workspace,
                                    size_t workspace_bytes, void* slots_bf16, void* dev_out, void* host_out_bf16,
                                    int32_t* status, void* stream) {
  using namespace b200moe;
  if (!w || !host_x_bf16 || !host_logits || !dev_x || !dev_logits || !dev_out || !host_out_bf16) return B200MOE_E_ARG;
  if (tokens < 1 || tokens > B200MOE_MAX_TOKENS) return B200MOE_E_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(dev_x, host_x_bf16, tokens * kH * 2, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return static_cast<int>(e);
  e = cudaMemcpyAsync(dev_logits, host_logits, tokens * w->num_experts * 4, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int r = b200moe_forward(w, dev_x, dev_logits, tokens, workspace, workspace_bytes, slots_bf16, dev_out, status, stream);
  if (r) return r;
  e = cudaMemcpyAsync(host_out_bf16, dev_out, tokens * kH * 2, cudaMemcpyDeviceToHost, s);
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}
