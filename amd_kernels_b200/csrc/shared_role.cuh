// The MXFP8 shared expert as a role of CTAs: both of its GEMMs (6144 -> SwiGLU -> I -> 6144, E4M3 x E4M3 with one E8M0 scale
// per 32 elements) by the last `ctas` CTAs of a launch whose other CTAs do the routed experts.
//
// Why inside another launch. At decode sizes the shared expert is 14.6 MB of weights against 7.5 MB for every routed expert
// that is hit, and a chain of its own (quantise, GEMM1 on 12 CTAs, GEMM2 on 48) is 30 us of latency: 17 + 15 us measured at 1
// token, with most SMs idle, in front of or behind kernels that fill the chip with one 170 KB CTA per SM. A side stream does
// not overlap them (whichever starts first holds the SMs) and costs four event calls on the host. As a role of 16 to 48 CTAs it
// runs beside the routed experts' weight stream, which is bound by HBM and does not miss those SMs.
//
// What bounds it: the thread that issues the MMAs (about 60 cycles per tcgen05 instruction, 48 K-tiles of 128 elements per
// unit), not the bytes. Unit = (block of bm tokens, weight tile of 128 rows); first all GEMM1 units, then all GEMM2 units,
// claimed in that order from a ticket. A GEMM2 unit waits -- bounded -- until the W13 tiles of its block are counted done;
// GEMM1 units never wait, and whoever claimed one is running, so the wait ends whichever CTAs of the launch are resident and
// whatever else runs on the device.
//
//   warp 0    producer (weights, tokens, token scales)     warp 1    MMA issue
//   warp 6    scale copies to tensor memory                warps 2-5 epilogue
#pragma once
#include "tc_host.cuh"
#include "tc_ptx.cuh"

namespace b200moe {

constexpr int kS1TilesK = kH / 128;  // 48 K-tiles of 128 elements in the shared expert's first GEMM
constexpr int kS2TilesK = kI / 128;  // 6 (or 12) in the second

struct SharedArgs {
  const uint8_t* w13t;  // tile records of both weights
  const uint8_t* w2t;
  const uint8_t* sfx8;  // input scale atoms [blocks][48][512]
  uint8_t* h8;          // GEMM1 out: E4M3 codes [rows][I]
  uint8_t* sfh8;        // GEMM1 out: scale atoms [blocks][I/128][512]
  __nv_bfloat16* out;   // bf16 [tokens][6144]
  int32_t* done;        // [blocks] finished GEMM1 tiles, zero at entry
  int32_t* ticket;      // units claimed so far, zero at entry
  int64_t tokens;
  int n_blocks, bm;     // dense blocks of bm = 16 / 32 / 64 / 128 tokens
  int stages;
  int ctas;             // 0: the launch has no such role
};

// What a launch needs to run the role, filled on the host (shared_plan in shared_tc.cu).
struct SharedPlan {
  CUtensorMap map_x, map_h;
  SharedArgs args;
};

struct SharedWorkspace {
  uint8_t *x8, *sfx8, *h8, *sfh8;
  size_t bytes;
  int bm;
  int64_t rows;
};
SharedWorkspace carve_shared(uint8_t* base, int64_t tokens);
int shared_plan(SharedPlan* plan, const uint8_t* w13t, const uint8_t* w2t, const uint8_t* codes8, int64_t code_rows,
                const SharedWorkspace& ws, void* out_bf16, int64_t tokens, int32_t* done, bool both);

// int32 words of a decode launch that belong to the role, zero at entry: finished GEMM1 tiles per block of tokens (at most 512
// tokens in blocks of 128), the last one its ticket
constexpr int kSharedDone = 8;
constexpr int kSharedMaxStages = 8;
constexpr int kSharedMaxSmem = 225 * 1024;  // opt-in limit of the kernels that carry the role
// shared memory: [stages x (record | tokens | scales)][epilogue staging]
__host__ __device__ inline int shared_stage_bytes(int bm) { return kTileRecordBytes + bm * 128 + 1024; }
__host__ __device__ inline int shared_epi_bytes(int bm) { return (bm < 64 ? bm : 64) * 136 * 4; }
static inline int shared_stages(int bm) { return bm == 128 ? 5 : bm == 64 ? 6 : 8; }
static inline int shared_smem_bytes(int bm) { return shared_stages(bm) * shared_stage_bytes(bm) + shared_epi_bytes(bm) + 1024; }

// A word that counts finished tiles: the low byte, signed (gemm12_kernel hands out its units above that).
__device__ __forceinline__ int tiles_done(int word) { return static_cast<int8_t>(word & 255); }

// Bounded wait for such a count in global memory (an acquire load).
__device__ __forceinline__ bool wait_count(const int32_t* counter, int target, volatile int* abort_flag, int32_t* status) {
  const uint64_t t0 = global_timer();
  uint32_t spins = 0;
  while (true) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
    if (tiles_done(v) >= target) return true;
    if ((++spins & 63u) == 0u) {
      if (*abort_flag) return false;
      if (global_timer() - t0 > wait_limit_ns()) {
        *abort_flag = 1;
        atomicExch(status, B200MOE_DEV_TIMEOUT);
        return false;
      }
    }
  }
}

// The units of a CTA whose work is handed out while it runs. One thread (the weight producer) claims a unit and puts it into a
// ring in shared memory; the other roles take the units from there in the same order. The barriers have count 1. An entry is
// written again kUnitRing units later: the producer is at most ceil(8 / 3) units ahead of the MMA thread (8 stages, units of at
// least 3), that one at most two ahead of the epilogue (two accumulators), and one unit is claimed ahead.
constexpr int kUnitRing = 16;
constexpr int kNoUnit = 0x7fffffff;  // beyond every list: the CTA is aborting
struct UnitRing {
  uint64_t* bar;
  volatile int* unit;
  __device__ __forceinline__ void put(uint32_t i, int u) const {
    unit[i % kUnitRing] = u;
    mbar_arrive(smem_u32(bar + i % kUnitRing));
  }
  __device__ __forceinline__ int get(uint32_t i, volatile int* abort_flag, int32_t* status) const {
    if (!mbar_wait(smem_u32(bar + i % kUnitRing), (i / kUnitRing) & 1u, abort_flag, status)) return kNoUnit;
    return unit[i % kUnitRing];
  }
};

// The barriers (bar_full, bar_empty, bar_sf: count 1 and at least a.stages long; bar_tfull[2] count 1; bar_tempty[2] count 128;
// bar_drain[2] count 1; those of `ring`) are initialised by the caller, tensor memory has at least 2 * bm + 64 columns, and the
// caller has passed its wait for the predecessor. `smem` is the 1024-byte aligned dynamic shared memory, `tiles` its 32-bit
// address.
__device__ __forceinline__ void shared_role(const SharedArgs& a, const CUtensorMap* map_x, const CUtensorMap* map_h,
                                            uint8_t* smem, uint32_t tiles, uint32_t tmem_base, uint64_t* bar_full,
                                            uint64_t* bar_empty, uint64_t* bar_sf, uint64_t* bar_tfull, uint64_t* bar_tempty,
                                            uint64_t* bar_drain, const UnitRing ring, volatile int* abort_v,
                                            int32_t* status) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bm = a.bm, ctas = a.ctas;
  const uint32_t stages = a.stages;
  const uint32_t b_off = kTileRecordBytes, sfb_off = b_off + bm * 128, stage_bytes = sfb_off + 1024;
  const int first = static_cast<int>(blockIdx.x) - (static_cast<int>(gridDim.x) - ctas);
  const int units1 = a.n_blocks * kW13Tiles, total = units1 + a.n_blocks * kW2Tiles;
  const uint32_t sfa_col = 2 * bm;  // 8 scale sets of (4 weight + 4 token) columns behind the two accumulators

  if (warp == 0) {
    if (lane == 0) {  // ------------------------------------------------ producer
      const uint32_t full0 = smem_u32(bar_full), empty0 = smem_u32(bar_empty);
      uint32_t it = 0, slot = 0, ph = 1u, base = tiles, full = full0, empty = empty0;
      bool ok = true;
      int u = atomicAdd(a.ticket, 1);
      ring.put(0, u);
      for (int mt = first; mt < kW2Tiles; mt += ctas)  // the CTAs share the GEMM2 weights' way into L2
        l2_prefetch_bulk(a.w2t + static_cast<int64_t>(mt) * kS2TilesK * kTileRecordBytes, kS2TilesK * kTileRecordBytes);
      for (uint32_t ui = 0; u < total && ok; ++ui) {
        int next = kNoUnit;
        const bool second = u >= units1;
        const int v = second ? u - units1 : u, tiles_m = second ? kW2Tiles : kW13Tiles;
        const int tiles_k = second ? kS2TilesK : kS1TilesK;
        const int b = v / tiles_m, mt = v % tiles_m;
        const uint8_t* w_src = (second ? a.w2t : a.w13t) + static_cast<int64_t>(mt) * tiles_k * kTileRecordBytes;
        const uint8_t* sf_src = (second ? a.sfh8 : a.sfx8) + static_cast<int64_t>(b) * tiles_k * kAtomBytes;
        if (second) {  // h of this block must be complete and visible to the copy engine
          if (!wait_count(a.done + b, kW13Tiles, abort_v, status)) { ok = false; break; }
          asm volatile("fence.proxy.async;" ::: "memory");
        }
        for (int kt = 0; kt < tiles_k; ++kt, ++it) {
          if (!mbar_wait(empty, ph, abort_v, status)) { ok = false; break; }
          // late in the unit, so that a CTA which is ahead gets more of them, and early enough to hide the atomic's way
          if (kt == tiles_k - 4) next = atomicAdd(a.ticket, 1);
          mbar_arrive_expect_tx(full, 128 * 128 + kAtomBytes + bm * 128 + kAtomBytes);
          bulk_load(base, w_src, 128 * 128 + kAtomBytes, full);
          tma_load_2d(base + b_off, second ? map_h : map_x, kt * 128, b * bm, full);
          bulk_load(base + sfb_off, sf_src, kAtomBytes, full);
          w_src += kTileRecordBytes;
          sf_src += kAtomBytes;
          if (++slot == stages) {
            slot = 0; ph ^= 1u; base = tiles; full = full0; empty = empty0;
          } else {
            base += stage_bytes; full += 8; empty += 8;
          }
        }
        if (!ok) break;
        ring.put(ui + 1, next);
        u = next;
      }
      if (!ok) drain_copies(bar_full, it, stages);
    }
  } else if (warp == 1) {
    {  // ------------------------------------------------ MMA issue
      // E4M3 x E4M3 (format 0), UE8M0 scales, M = 128 weight rows, N = bm tokens; scale byte k of a row's cell for MMA k
      const uint32_t idesc = (static_cast<uint32_t>(bm >> 3) << 17) | (1u << 23) | (8u << 24);
      const uint32_t sf0 = smem_u32(bar_sf), empty0 = smem_u32(bar_empty);
      uint32_t slot = 0, ph = 0, sfset = 0;
      uint32_t lo = tiles >> 4, sf = sf0, empty = empty0;
      bool ok = true;
      for (uint32_t ui = 0; ok; ++ui) {
        const int u = __shfl_sync(0xffffffffu, ring.get(ui, abort_v, status), 0);
        if (u >= total) break;
        const int tiles_k = u >= units1 ? kS2TilesK : kS1TilesK;
        const uint32_t acc = ui & 1u, aph = (ui >> 1) & 1u;
        if (!warp_wait(smem_u32(bar_tempty + acc), aph ^ 1u, abort_v, status)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * bm;
        for (int kt = 0; kt < tiles_k; ++kt) {
          if (!warp_wait(sf, ph, abort_v, status)) { ok = false; break; }
          tc_fence_after();
          const uint32_t t_sfa = tmem_base + sfa_col + 8u * sfset, t_sfb = t_sfa + 4u;
          const uint32_t w_lo = lo, x_lo = lo + (b_off >> 4);
          if (elect_one()) {
            tc_mma_mxf8_lo<2>(d_tmem, w_lo, x_lo, idesc, t_sfa, t_sfb, static_cast<uint32_t>(kt != 0));
            tc_mma_mxf8_lo<1>(d_tmem, w_lo + 2, x_lo + 2, idesc | (1u << 29) | (1u << 4), t_sfa, t_sfb);
            tc_mma_mxf8_lo<1>(d_tmem, w_lo + 4, x_lo + 4, idesc | (2u << 29) | (2u << 4), t_sfa, t_sfb);
            tc_mma_mxf8_lo<1>(d_tmem, w_lo + 6, x_lo + 6, idesc | (3u << 29) | (3u << 4), t_sfa, t_sfb);
            tc_commit(empty);
          }
          __syncwarp();
          sfset = (sfset + 1u) & (kSharedMaxStages - 1);
          if (++slot == stages) {
            slot = 0; ph ^= 1u; lo = tiles >> 4; sf = sf0; empty = empty0;
          } else {
            lo += stage_bytes >> 4; sf += 8; empty += 8;
          }
        }
        if (ok && elect_one()) tc_commit(smem_u32(bar_tfull + acc));
      }
      if (__any_sync(0xffffffffu, *abort_v != 0) && elect_one()) drain_tcgen05(smem_u32(bar_drain));
    }
  } else if (warp == 6) {
    {  // ------------------------------------------------ scale copies: shared memory -> tensor memory
      const uint32_t full0 = smem_u32(bar_full), sf0 = smem_u32(bar_sf);
      uint32_t slot = 0, ph = 0, sfset = 0;
      uint32_t lo = tiles >> 4, full = full0, sf = sf0;
      bool ok = true;
      for (uint32_t ui = 0; ok; ++ui) {
        const int u = __shfl_sync(0xffffffffu, ring.get(ui, abort_v, status), 0);
        if (u >= total) break;
        const int tiles_k = u >= units1 ? kS2TilesK : kS1TilesK;
        for (int kt = 0; kt < tiles_k; ++kt) {
          if (!warp_wait(full, ph, abort_v, status)) { ok = false; break; }
          tc_fence_after();
          const uint32_t t_sfa = tmem_base + sfa_col + 8u * sfset;
          if (elect_one()) {
            tc_cp_scales_lo(t_sfa, lo + ((128 * 128) >> 4));
            tc_cp_scales_lo(t_sfa + 4, lo + (sfb_off >> 4));
            tc_commit(sf);
          }
          __syncwarp();
          sfset = (sfset + 1u) & (kSharedMaxStages - 1);
          if (++slot == stages) {
            slot = 0; ph ^= 1u; lo = tiles >> 4; full = full0; sf = sf0;
          } else {
            lo += stage_bytes >> 4; full += 8; sf += 8;
          }
        }
      }
      if (__any_sync(0xffffffffu, *abort_v != 0) && elect_one()) drain_tcgen05(smem_u32(bar_drain + 1));
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const int q = warp & 3;
    const int et = threadIdx.x - 64;
    float* stage_f = reinterpret_cast<float*>(smem + stages * stage_bytes);
    for (uint32_t ui = 0;; ++ui) {
      const int u = ring.get(ui, abort_v, status);
      const bool second = u >= units1;
      const int v = second ? u - units1 : u, tiles_m = second ? kW2Tiles : kW13Tiles;
      const int b = v / tiles_m, mt = v % tiles_m;
      const uint32_t acc = ui & 1u, aph = (ui >> 1) & 1u;
      const int64_t row0 = static_cast<int64_t>(b) * bm;
      if (!epilogue_all(u < total && mbar_wait(smem_u32(bar_tfull + acc), aph, abort_v, status), 1u)) break;
      tc_fence_after();
      const uint32_t t_acc = tmem_base + acc * bm + (static_cast<uint32_t>(q * 32) << 16);
      const int row_floats = second ? 132 : 136, cols = min(bm, second ? 32 : 64);
      float* mine = second ? stage_f + q * 32 + lane : stage_f + (q >> 1) * 68 + (q & 1) * 32 + lane;
#pragma unroll 1
      for (int c0 = 0; c0 < bm; c0 += cols) {
#pragma unroll 1
        for (int cc = 0; cc < cols; cc += 16) {
          uint32_t t16[16];
          tc_ld16(t_acc + c0 + cc, t16);
#pragma unroll
          for (int j = 0; j < 16; ++j) mine[(cc + j) * row_floats] = __uint_as_float(t16[j]);
        }
        if (c0 + cols >= bm) {  // accumulator fully read: hand it back to the MMA thread
          tc_fence_before();
          mbar_arrive(smem_u32(bar_tempty + acc));
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (!second) {
          // one thread = one (token, 32-column group): SwiGLU-OAI, block maximum, E8M0 scale, 32 E4M3 codes
          for (int item = et; item < 2 * cols; item += 128) {
            const int j = item >> 1, g = item & 1;
            const float4* src = reinterpret_cast<const float4*>(stage_f + j * 136 + g * 68);
            float h[32];
            float amax = 0.0f;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float4 gv = src[k], uv = src[8 + k];
              h[4 * k + 0] = swiglu_oai(gv.x, uv.x);
              h[4 * k + 1] = swiglu_oai(gv.y, uv.y);
              h[4 * k + 2] = swiglu_oai(gv.z, uv.z);
              h[4 * k + 3] = swiglu_oai(gv.w, uv.w);
            }
#pragma unroll
            for (int k = 0; k < 32; ++k) amax = fmaxf(amax, fabsf(h[k]));
            const int sc = mxfp8_scale(amax);
            const float inv = __uint_as_float(static_cast<uint32_t>(254 - sc) << 23);
            uint32_t words[8];
#pragma unroll
            for (int wd = 0; wd < 8; ++wd)
              words[wd] = cvt_e4m3x2(h[4 * wd] * inv, h[4 * wd + 1] * inv) |
                          (cvt_e4m3x2(h[4 * wd + 2] * inv, h[4 * wd + 3] * inv) << 16);
            const int grp = 2 * mt + g, n = c0 + j;
            uint4* dst = reinterpret_cast<uint4*>(a.h8 + (row0 + n) * kI + grp * 32);
            dst[0] = make_uint4(words[0], words[1], words[2], words[3]);
            dst[1] = make_uint4(words[4], words[5], words[6], words[7]);
            a.sfh8[(static_cast<int64_t>(b) * kS2TilesK + (grp >> 2)) * kAtomBytes + atom_offset(n, grp & 3)] =
                static_cast<uint8_t>(sc);
          }
          // this thread's h stores: ordered for the copy engine and visible device-wide before the count moves
          asm volatile("fence.proxy.async;" ::: "memory");
          __threadfence();
        } else {
          // a warp writes one token's 128 output columns as 256 contiguous bytes
          for (int item = et; item < cols * 32; item += 128) {
            const int j = item >> 5, seg = item & 31;
            const int64_t row = row0 + c0 + j;
            if (row < a.tokens) {
              const float4 x4 = *reinterpret_cast<const float4*>(stage_f + j * 132 + seg * 4);
              const __nv_bfloat162 p0 = __floats2bfloat162_rn(x4.x, x4.y), p1 = __floats2bfloat162_rn(x4.z, x4.w);
              uint2 packed;
              packed.x = *reinterpret_cast<const uint32_t*>(&p0);
              packed.y = *reinterpret_cast<const uint32_t*>(&p1);
              *reinterpret_cast<uint2*>(a.out + row * kH + mt * 128 + seg * 4) = packed;
            }
          }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
      }
      if (!second && et == 0) atomicAdd(a.done + b, 1);  // one more GEMM1 tile of block b is complete
    }
  }
}

}  // namespace b200moe
