// Router GEMM on the tensor cores for prefill sizes: bf16 activations x the fp32 gate carried as three bf16 terms
// (hi = RN(w), mid = RN(w - hi), lo = RN(w - hi - mid), the split of the reference's router,
// amd_kernels/moe/mxfp4_h6144_i768_e128_top4/router_gemm.py:32-44), tcgen05.mma kind::f16 with fp32 accumulators in tensor
// memory. Output: the split-K partials fp32 [S][T][E] the top-4 kernel adds in split order, the layout b200moe_router_gemm
// writes on the CUDA cores.
//
// A unit is (block of 128 tokens, K split): the token block is the 128-row M operand (TMA, 128-byte swizzle; rows past T
// are filled with zeros by the copy engine), the 128 experts are N, and each 64-element K step issues four K = 16 MMAs per
// gate term (hi, mid, lo in turn) into one accumulator, so a partial is the fp32 sum of exact bf16 products.
//
//   warp 0    producer: one thread, four tile loads per stage (tokens, gate hi / mid / lo)
//   warp 1    allocates tensor memory and issues the MMAs
//   warps 2-5 epilogue: thread = token row (TMEM lane), 128 logits -> partials[s][t][0..E)
//   QUANT: warps 6-13 quantise the token tile while it is in shared memory (the layer call and the prepared input need x in MXFP4
//   and, for the shared expert, in MXFP8): two groups of four warps take the pairs of K steps in turn, a thread owns one row, whose
//   128 values of a pair make 64 bytes of E2M1 codes, 128 of E4M3 codes and two words of scales, in whole 32-byte sectors.
//
// Why the quantisers are here. Alone they read x again: 201 of 361 MB at 16384 tokens, behind a GEMM that leaves HBM idle. One pass
// is bound by HBM (x in, codes out), the GEMM's 768 tensor cycles per K step run under it. Measured, router GEMM + both quantisers /
// one kernel, us: 12 + 7 -> 13.5 at 777 tokens, 18 + 10 -> 23 at 2048, 39 + 32 -> 61 at 8191, 72 + 60 -> 115 at 16384. Without
// the quantisers' arithmetic the kernel takes 80 us there, without their stores 86: both operands of a 128 x 128 x 16 MMA come from
// shared memory at its full rate, beside the tiles that arrive. Two token blocks per unit (half the gate traffic), and asking for x
// a kilobyte of a row at a time through L2, measured the same.
#include "tc_host.cuh"
#include "tc_ptx.cuh"

namespace b200moe {

struct RouterCfg {
  static constexpr int kStages = 3;
  // A "landed" barrier per K step modulo 12, not per stage: the quantising groups take the pairs of steps in turn, and a group must
  // see every phase of a barrier that it waits on (12: the steps of one group, modulo 4, that share a stage, modulo 3).
  static constexpr int kFullBars = 12;
  static constexpr int kTileBytes = 128 * 128;            // 128 rows x 64 bf16
  static constexpr int kStageBytes = 4 * kTileBytes;      // tokens, gate hi, mid, lo
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024;
  static constexpr int kThreads = 192, kQuantThreads = 192 + 256;
  static constexpr int kTmemCols = 256;                   // two accumulators of 128 columns
  static constexpr int kKSteps = kH / 64;                 // 96 K steps of 64 elements over the hidden size
};

__device__ __forceinline__ void tc_mma_bf16_lo(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .b64 da, db;\n.reg .pred p;\nmov.b64 da, {%1, %5};\nmov.b64 db, {%2, %5};\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}\n" ::"r"(d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(kOperandDescHi)
      : "memory");
}

// gate fp32 [E][6144] -> three bf16 terms [3][128][6144]; rows from E on are zero
__global__ void __launch_bounds__(256) split_gate_kernel(const float* __restrict__ gate, int num_experts,
                                                         __nv_bfloat16* __restrict__ out) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<int64_t>(kMaxE) * kH) return;
  const int e = static_cast<int>(i / kH);
  float w = e < num_experts ? gate[i] : 0.0f;
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const __nv_bfloat16 t = __float2bfloat16_rn(w);
    out[static_cast<int64_t>(p) * kMaxE * kH + i] = t;
    w -= __bfloat162float(t);  // exact: the remainder of a round-to-nearest fits fp32
  }
}

// 32 values of a row (bf16, 64 bytes): the largest magnitude
__device__ __forceinline__ float block_amax(const uint4 (&raw)[4]) {
  float amax = 0.0f;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint32_t r[4] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      amax = fmaxf(amax, fmaxf(fabsf(__uint_as_float(r[j] << 16)), fabsf(__uint_as_float(r[j] & 0xffff0000u))));
  }
  return amax;
}
// Always 0, known once every lane has its two values. An arrival that frees a shared-memory stage has to depend on what was loaded
// from it: loads and arrivals of a warp are not executed in order, and a vote on the loads' results is what holds the arrival back.
__device__ __forceinline__ uint32_t landed(float a, float b) {
  uint32_t any;
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.lt.f32 p, %1, 0f00000000;\nsetp.lt.or.f32 p, %2, 0f00000000, p;\n"
      "vote.sync.any.pred q, p, 0xffffffff;\nselp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(any)
      : "f"(a), "f"(b)
      : "memory");
  return any;
}
__device__ __forceinline__ void store_sector(void* p, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]),
               "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// Where the quantised rows go: MXFP4 row-major, and (q8.codes may be null) MXFP8.
struct RouterQuant {
  uint8_t *codes4, *scales4;
  QuantRow8 q8;
};

template <bool QUANT>
__global__ void __launch_bounds__(QUANT ? RouterCfg::kQuantThreads : RouterCfg::kThreads, 1)
    router_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_g,
                     float* __restrict__ partials, int64_t tokens, int num_experts, int splits, int32_t* status,
                     const RouterQuant rq) {
  using C = RouterCfg;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[C::kFullBars];
  __shared__ __align__(8) uint64_t bar_empty[C::kStages];
  __shared__ __align__(8) uint64_t bar_tfull[2];
  __shared__ __align__(8) uint64_t bar_tempty[2];
  __shared__ __align__(8) uint64_t bar_drain;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tiles = (smem_u32(smem_raw) + 1023u) & ~1023u;
  volatile int* abort_v = &abort_flag;
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < C::kFullBars; ++s) mbar_init(smem_u32(&bar_full[s]), 1);
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(smem_u32(&bar_empty[s]), QUANT ? 1 + 4 : 1);  // the MMAs' commit (and the warps that quantise the step)
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&bar_tfull[a]), 1);
      mbar_init(smem_u32(&bar_tempty[a]), 128);
    }
    mbar_init(smem_u32(&bar_drain), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                 "r"(static_cast<uint32_t>(C::kTmemCols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  pdl_wait();

  const int total_units = static_cast<int>((tokens + 127) / 128) * splits;
  const int steps = C::kKSteps / splits;  // K steps of one split

  if (warp == 0) {
    if (lane == 0) {  // ------------------------------------------------ producer
      uint32_t it = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < total_units && ok; u += gridDim.x) {
        const int tb = u / splits, sp = u % splits;
        for (int i = 0; i < steps; ++i, ++it) {
          const uint32_t s = it % C::kStages, ph = (it / C::kStages) & 1u;
          if (!mbar_wait(smem_u32(&bar_empty[s]), ph ^ 1u, abort_v, status)) { ok = false; break; }
          const uint32_t full = smem_u32(&bar_full[it % C::kFullBars]), base = tiles + s * C::kStageBytes;
          const int kbyte = (sp * steps + i) * 128;
          mbar_arrive_expect_tx(full, C::kStageBytes);
          tma_load_2d(base, &map_x, kbyte, tb * 128, full);
#pragma unroll
          for (int p = 0; p < 3; ++p) tma_load_2d(base + (1 + p) * C::kTileBytes, &map_g, kbyte, p * kMaxE, full);
        }
      }
      if (!ok) drain_copies(bar_full, it, C::kFullBars);
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------------- MMA issue
    // bf16 x bf16 -> fp32, both operands K-major, M = 128 token rows, N = 128 experts
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(128 >> 3) << 17) |
                                (static_cast<uint32_t>(128 >> 4) << 24);
    uint32_t it = 0, ui = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < total_units && ok; u += gridDim.x, ++ui) {
      const uint32_t acc = ui & 1u, aph = (ui >> 1) & 1u;
      if (!warp_wait(smem_u32(&bar_tempty[acc]), aph ^ 1u, abort_v, status)) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + acc * 128u;
      for (int i = 0; i < steps; ++i, ++it) {
        const uint32_t s = it % C::kStages, ph = (it / C::kFullBars) & 1u;
        if (!warp_wait(smem_u32(&bar_full[it % C::kFullBars]), ph, abort_v, status)) { ok = false; break; }
        tc_fence_after();
        const uint32_t x_lo = (tiles + s * C::kStageBytes) >> 4;
        if (elect_one()) {
#pragma unroll
          for (int k4 = 0; k4 < 4; ++k4) {  // 16 K-elements = 32 bytes (descriptor + 2) per MMA
#pragma unroll
            for (int p = 1; p <= 3; ++p)
              tc_mma_bf16_lo(d_tmem, x_lo + 2 * k4, x_lo + p * (C::kTileBytes >> 4) + 2 * k4, kIdesc,
                             static_cast<uint32_t>(i != 0 || k4 != 0 || p != 1));
          }
          tc_commit(smem_u32(&bar_empty[s]));
          if (i == steps - 1) tc_commit(smem_u32(&bar_tfull[acc]));
        }
        __syncwarp();
      }
    }
    if (__any_sync(0xffffffffu, *abort_v != 0) && elect_one()) drain_tcgen05(smem_u32(&bar_drain));
  } else if (QUANT && warp >= 6) {
    // -------------------------------------------------------------------- quantisers (warps 6..13)
    const uint32_t group = static_cast<uint32_t>(warp - 6) >> 2;
    const int tr = ((warp - 6) & 3) * 32 + lane;
    const uint8_t* tile = smem_raw + (tiles - smem_u32(smem_raw)) + tr * 128;
    uint32_t it = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < total_units && ok; u += gridDim.x) {
      const int64_t t = static_cast<int64_t>(u / splits) * 128 + tr;
      const int step0 = u % splits * steps;
      for (int i = 0; i < steps && ok; i += 2, it += 2) {  // (steps are even: the host's rule)
        if (((it >> 1) & 1u) != group) continue;
        const int atom = (step0 + i) >> 1;  // 128 elements: four blocks
        uint32_t sc4 = 0, sc8 = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t s = (it + h) % C::kStages, ph = ((it + h) / C::kFullBars) & 1u;
          if (!warp_wait(smem_u32(&bar_full[(it + h) % C::kFullBars]), ph, abort_v, status)) {
            ok = false;
            break;
          }
          uint4 raw[2][4];
#pragma unroll
          for (int c = 0; c < 8; ++c)
            raw[c >> 2][c & 3] = *reinterpret_cast<const uint4*>(tile + s * C::kStageBytes + ((c ^ (tr & 7)) << 4));
          const float amax[2] = {block_amax(raw[0]), block_amax(raw[1])};
          const uint32_t zero = landed(amax[0], amax[1]);
          if (lane == 0) mbar_arrive(smem_u32(&bar_empty[s]) + zero);  // the rows sit in registers
          uint32_t o4[8];
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const int e = quark_even_e8m0(amax[b]), e8 = mxfp8_scale(amax[b]);
            const float inv = __uint_as_float(static_cast<uint32_t>(254 - e) << 23);  // 2^(127-e), exact
            const float inv8 = __uint_as_float(static_cast<uint32_t>(254 - e8) << 23);
            sc4 |= static_cast<uint32_t>(e) << (8 * (2 * h + b));
            sc8 |= static_cast<uint32_t>(e8) << (8 * (2 * h + b));
            uint32_t o8[8];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const uint32_t r[4] = {raw[b][c].x, raw[b][c].y, raw[b][c].z, raw[b][c].w};
              float v[8];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                v[2 * j] = __uint_as_float(r[j] << 16);
                v[2 * j + 1] = __uint_as_float(r[j] & 0xffff0000u);
              }
              uint32_t packed = 0;
#pragma unroll
              for (int j = 0; j < 4; ++j) packed |= cvt_e2m1x2(v[2 * j] * inv, v[2 * j + 1] * inv) << (8 * j);
              o4[4 * b + c] = packed;
              o8[2 * c] = cvt_e4m3x2(v[0] * inv8, v[1] * inv8) | (cvt_e4m3x2(v[2] * inv8, v[3] * inv8) << 16);
              o8[2 * c + 1] = cvt_e4m3x2(v[4] * inv8, v[5] * inv8) | (cvt_e4m3x2(v[6] * inv8, v[7] * inv8) << 16);
            }
            if (rq.q8.codes != nullptr && t < tokens) store_sector(rq.q8.codes + t * kH + atom * 128 + h * 64 + b * 32, o8);
          }
          if (t < tokens) store_sector(rq.codes4 + t * (kH / 2) + atom * 64 + h * 32, o4);
        }
        if (ok && t < tokens) {
          *reinterpret_cast<uint32_t*>(rq.scales4 + t * (kH / 32) + atom * 4) = sc4;
          if (rq.q8.codes != nullptr) rq.q8.store_scales(t, atom, sc8);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const int q = warp & 3;
    const int tr = q * 32 + lane;
    uint32_t ui = 0;
    for (int u = blockIdx.x; u < total_units; u += gridDim.x, ++ui) {
      const int tb = u / splits, sp = u % splits;
      const uint32_t acc = ui & 1u, aph = (ui >> 1) & 1u;
      if (!epilogue_all(mbar_wait(smem_u32(&bar_tfull[acc]), aph, abort_v, status), 1u)) break;
      tc_fence_after();
      const int64_t t = static_cast<int64_t>(tb) * 128 + tr;
      float* dst = partials + (static_cast<int64_t>(sp) * tokens + t) * num_experts;
      const uint32_t t_acc = tmem_base + acc * 128u + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t v[32];
        tc_ld32(t_acc + 32 * c, v);
        if (c == 3) {  // accumulator read: hand it back to the MMA warp
          tc_fence_before();
          mbar_arrive(smem_u32(&bar_tempty[acc]));
        }
        if (t < tokens) {
          if (num_experts == kMaxE) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
              *reinterpret_cast<uint4*>(dst + 32 * c + 4 * k) = make_uint4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
          } else {
#pragma unroll
            for (int k = 0; k < 32; ++k)
              if (32 * c + k < num_experts) dst[32 * c + k] = __uint_as_float(v[k]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(C::kTmemCols))
                 : "memory");
  }
}

int set_wait_limit_router(unsigned long long ns) { return set_wait_limit_here(ns); }

}  // namespace b200moe

extern "C" int b200moe_router_split_gate(const float* gate, int num_experts, void* split_bf16, void* stream) {
  using namespace b200moe;
  if (!gate || !split_bf16 || num_experts < 1 || num_experts > kMaxE) return B200MOE_E_ARG;
  if (misaligned(split_bf16, 16)) return B200MOE_E_ALIGN;
  const int64_t n = static_cast<int64_t>(kMaxE) * kH;
  B200MOE_LAUNCH_PLAIN(split_gate_kernel, static_cast<unsigned>((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream),
                       gate, num_experts, static_cast<__nv_bfloat16*>(split_bf16));
  return 0;
}

namespace b200moe {
template <bool QUANT>
static int launch_router_tc(const void* x_bf16, const void* gate_split_bf16, int64_t tokens, int num_experts, int splits,
                            float* partials, const RouterQuant& rq, int32_t* status, void* stream) {
  using C = RouterCfg;
  if (!x_bf16 || !gate_split_bf16 || !partials || !status || tokens < 0 || num_experts < 1 || num_experts > kMaxE)
    return B200MOE_E_ARG;
  if (splits < 1 || C::kKSteps % splits) return B200MOE_E_ARG;
  if (misaligned(x_bf16, 16) || misaligned(gate_split_bf16, 16) || misaligned(partials, 16)) return B200MOE_E_ALIGN;
  if (tokens == 0) return 0;
  CUtensorMap mx, mg;
  int r = make_map(&mx, x_bf16, kH * 2, static_cast<uint64_t>(tokens), 128);
  if (r) return r;
  if ((r = make_map(&mg, gate_split_bf16, kH * 2, 3 * kMaxE, 128))) return r;
  static PerDeviceOnce once;
  const int rc = once.run([] {
    return static_cast<int>(cudaFuncSetAttribute(router_tc_kernel<QUANT>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
  });
  if (rc) return rc;
  const int64_t units = (tokens + 127) / 128 * splits;
  const int grid = static_cast<int>(units < sm_count() ? units : sm_count());
  B200MOE_LAUNCH(router_tc_kernel<QUANT>, grid, QUANT ? C::kQuantThreads : C::kThreads, C::kSmemBytes,
                 static_cast<cudaStream_t>(stream), mx, mg, partials, tokens, num_experts, splits, status, rq);
  return 0;
}

int quant_rows(const void* x_bf16, int64_t tokens, uint8_t* codes, uint8_t* scales, void* stream);
int quant_rows_both(const void* x_bf16, int64_t tokens, uint8_t* codes, uint8_t* scales, uint8_t* codes8, uint8_t* scales8,
                    uint8_t* atoms8, int bm8, void* stream);

// The router GEMM and the input quantisers (codes8 may be null: MXFP4 only). One pass over x from 257 tokens on; below, the 16 to 32
// CTAs of the GEMM are too few to quantise (the layer at 128 / 200 / 256 tokens, two kernels / one: 158 / 160, 175 / 177, 185 / 188 us;
// 227 / 225 at 400). Two kernels also where an output is not aligned to the 32-byte sectors that the one-pass form stores, or a split
// has an odd number of K steps.
constexpr int64_t kOnePassFrom = 257;
int router_tc_quant(const void* x_bf16, const void* gate_split_bf16, int64_t tokens, int num_experts, int splits, float* partials,
                    uint8_t* codes4, uint8_t* scales4, uint8_t* codes8, uint8_t* scales8, uint8_t* atoms8, int bm8, int32_t* status,
                    void* stream) {
  if (!codes4 || !scales4 || (codes8 && !scales8 && !atoms8)) return B200MOE_E_ARG;
  const bool one_pass = tokens >= kOnePassFrom && splits >= 1 && RouterCfg::kKSteps % (2 * splits) == 0 && !misaligned(codes4, 32) &&
                        !misaligned(codes8, 32) && !misaligned(scales4, 4) && !misaligned(scales8, 4) && !misaligned(atoms8, 16);
  if (one_pass) {
    const int shift = bm8 == 16 ? 4 : bm8 == 32 ? 5 : bm8 == 64 ? 6 : 7;
    return launch_router_tc<true>(x_bf16, gate_split_bf16, tokens, num_experts, splits, partials,
                                  RouterQuant{codes4, scales4, QuantRow8{codes8, scales8, atoms8, shift}}, status, stream);
  }
  const int r = b200moe_router_gemm_tc(x_bf16, gate_split_bf16, tokens, num_experts, splits, partials, status, stream);
  if (r) return r;
  return codes8 ? quant_rows_both(x_bf16, tokens, codes4, scales4, codes8, scales8, atoms8, bm8, stream)
                : quant_rows(x_bf16, tokens, codes4, scales4, stream);
}
}  // namespace b200moe

extern "C" int b200moe_router_gemm_tc(const void* x_bf16, const void* gate_split_bf16, int64_t tokens, int num_experts,
                                      int splits, float* partials, int32_t* status, void* stream) {
  return b200moe::launch_router_tc<false>(x_bf16, gate_split_bf16, tokens, num_experts, splits, partials, b200moe::RouterQuant{},
                                          status, stream);
}
