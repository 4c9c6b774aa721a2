// The MXFP8 shared expert at prefill sizes, on CTA pairs: tcgen05.mma.cta_group::2 kind::mxf8f6f4 with M = 256 token rows (two
// blocks of 128) x N = 256 weight rows (two weight tiles) x K = 32 per instruction. Same operands, records and results (bit for
// bit) as shared_gemm_kernel<MODE, 128>, which keeps the weight tile as the 128-row operand.
//
// What bounds it: operand bytes into shared memory. A 128-element K-tile of a 128 x 128 unit on one CTA needs 33 KB for 256
// cycles of tensor time, and an SM takes in about 64 bytes per cycle (half of the tensor rate at best); in a pair each CTA
// stages its own 128 token rows and half of the weight rows, 33.5 KB for 512 cycles. The dense blocks leave no odd half inside
// the work (only the last block of an odd count runs with an idle partner).
//
// Unit = (pair of token blocks) x (pair of weight tiles). Two rings, as in gemm1_wide_kernel: 6 stages of codes (MODE 3: 4), and 8
// slots of scales that travel ahead of them, so that the MMA warp waits for codes only.
//
//   warp 0      code producer (both CTAs): TMA of the CTA's 128 token rows and of its weight tile, counted on the leader's barrier
//   warp 1      tensor memory (both CTAs); in the leader it issues the MMAs for both, the whole warp around one elected lane
//   warp 2      leader: copies the scales into tensor memory in both CTAs, in the same way
//   warp 3      scale producer (both CTAs): the CTA's token scales, the scales of both weight tiles
//   warps 4-11  epilogue (both CTAs): thread = one token row. MODE 1: 128 accumulator values into registers, the accumulator is
//               handed back, then SwiGLU-OAI + E4M3 requantisation, thread-local. MODE 2 and 3: the values are read in two halves
//               and rounded to bf16, 64 registers a row, before it is handed back; then through a strip of shared memory per
//               warp so that eight or sixteen lanes store full lines of a row
// Measured, one-CTA kernel / pairs, both GEMMs and the scale layout, cold L2: 348 / 192 us at 16384 tokens, 173 / 99 at 8191, 93 / 67
// at 4096. Counters at 8192 tokens, before the issuing warps elected a lane: tensor pipe 70 % busy in the first GEMM, DRAM 11 %.
// Cycles of the MMA thread per K-tile at 16384 tokens (512 are tensor time), read from the clock in a build of that form: 690, of
// which the four MMAs and the looks at the next stage's barriers 350, the stage release 74, waiting for scales 190, for codes 55.
// Before the looks, with two plain waits, two commits per release and the accumulator handed back by a cluster-scope release, it was
// 750 and the whole 251 us.
// MODE 3 is MODE 2 for a call that hands out neither the shared rows nor anything but the sum: its epilogue has the shared value
// of a (token, column) in a register and adds the four slots in front of it, out = bf16((((0 + s0) + s1) + s2) + s3 + bf16(shared)),
// the slot reduce's sum bit for bit. So the shared rows are never written nor read back, and the slot reduce's traffic (40 KB a
// token, HBM bound) runs under this GEMM's arithmetic and not behind it. Each epilogue thread keeps 16 to 32 16-byte slot loads in
// flight, a batch ahead and across units, so the rings give shared memory back (four stages) for the L1 lines those loads need.
// Measured, second GEMM + slot reduce / MODE 3: 77 + 166 -> 168 us at 16384 tokens (1.05 GB; its bytes alone take 160 at the copy
// rate), I = 1536 41 + 42 -> 54 at 4096.
// 12 warps start with 168 registers; the issuing warpgroup drops to 72, the epilogue's rise to 216 (4 x 72 + 8 x 216 = 12 x 168:
// the exchange must balance inside what the CTA was given at launch). MODE 3 spills 24 bytes a thread (stores; 60 bytes of loads),
// MODE 1 and 2 nothing.
#include "shared_role.cuh"
#include "tc_pair.cuh"

namespace b200moe {

template <int MODE>
struct SharedPairCfg {
  static constexpr int kTilesM = MODE == 1 ? kW13Tiles : kW2Tiles;
  static constexpr int kTilePairs = kTilesM / 2;
  static constexpr int kTilesK = MODE == 1 ? kS1TilesK : kS2TilesK;
  static constexpr int kStages = MODE == 3 ? 4 : 6; // code ring
  static constexpr int kSfStages = 8;               // scale ring = scale sets in tensor memory
  static constexpr int kTokOff = 0;                 // this CTA's 128 token rows x 128 bytes
  static constexpr int kWOff = 128 * 128;           // its 128 weight rows: tile 2 * tp + rank
  static constexpr int kStageBytes = 2 * 128 * 128;
  static constexpr int kSfRingOff = kStages * kStageBytes;
  static constexpr int kSfTokOff = 0, kSfWLoOff = kAtomBytes, kSfWHiOff = 2 * kAtomBytes;  // inside a scale slot
  static constexpr int kSfSlotBytes = 3 * kAtomBytes;
  static constexpr int kStripOff = kSfRingOff + kSfStages * kSfSlotBytes;
  // epilogue of MODE 2 and 3, a warp's 32 rows x 128 columns in four parts: 16 rows x 64 columns, 8 lanes to a row's 128 bytes, or 8
  // rows x 128 columns, 16 lanes to 256 bytes. The longer piece reads the slots faster (MODE 3: 187 -> 168 us at 16384 tokens), the
  // shorter one stores the rows alone faster (35.5 / 37.0 us at 8191).
  static constexpr int kLanesPerRow = MODE == 3 ? 16 : 8, kPartRows = 128 / kLanesPerRow;
  static constexpr int kStripRow = kLanesPerRow * 16 + 16, kStripBytes = kPartRows * kStripRow;  // + 16: eight lanes' writes hit all banks
  static constexpr int kSmemBytes = kStripOff + (MODE >= 2 ? 8 * kStripBytes : 0) + 1024;
  static constexpr int kThreads = 32 * 12;
  static constexpr int kSfCol = 256;                // tensor memory: 256 accumulator columns, then 8 sets of 16
  static constexpr int kTmemCols = 512;
};
template <int MODE>
constexpr bool shared_pair_fits() {
  using C = SharedPairCfg<MODE>;
  static_assert(C::kSmemBytes <= 227 * 1024, "shared memory");
  static_assert(C::kSfStages >= C::kStages, "a scale set is free once the code stage is");
  return true;
}
static_assert(shared_pair_fits<1>() && shared_pair_fits<2>() && shared_pair_fits<3>());

__device__ __forceinline__ void tc_mma_mxf8_pair(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t sfa,
                                                 uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .b64 da, db;\n.reg .pred p;\nmov.b64 da, {%1, %7};\nmov.b64 db, {%2, %7};\nsetp.ne.b32 p, %6, 0;\n"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], da, db, %3, [%4], [%5], p;\n}\n" ::"r"(d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate), "n"(kOperandDescHi)
      : "memory");
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(SharedPairCfg<MODE>::kThreads, 1)
    shared_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_sfx,
                       const __grid_constant__ CUtensorMap map_wc, const __grid_constant__ CUtensorMap map_ws, int n_blocks,
                       int64_t tokens, uint8_t* __restrict__ h8, uint8_t* __restrict__ sfh8,
                       const __nv_bfloat16* __restrict__ slots, __nv_bfloat16* __restrict__ out, int32_t* status) {
  using C = SharedPairCfg<MODE>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[C::kStages];     // leader: both CTAs' codes of the stage have landed
  __shared__ __align__(8) uint64_t bar_empty[C::kStages];    // in each CTA: the MMAs that read the stage have completed
  __shared__ __align__(8) uint64_t bar_sfull[C::kSfStages];  // leader: both CTAs' scales of the slot have landed
  __shared__ __align__(8) uint64_t bar_sf[C::kSfStages];     // in each CTA: they have been copied to tensor memory
  __shared__ __align__(8) uint64_t bar_tfull;                // in each CTA: the unit's accumulator is complete
  __shared__ __align__(8) uint64_t bar_tempty;               // leader: both CTAs' epilogues have read it
  __shared__ __align__(8) uint64_t bar_drain[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const uint32_t tiles = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sf_ring = tiles + C::kSfRingOff;
  volatile int* abort_v = &abort_flag;
  pdl_launch_dependents();

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int j = 0; j < C::kSfStages; ++j) {
      mbar_init(smem_u32(&bar_sfull[j]), 1);
      mbar_init(smem_u32(&bar_sf[j]), 1);
    }
    mbar_init(smem_u32(&bar_tfull), 1);
    mbar_init(smem_u32(&bar_tempty), 16);  // one arrival per epilogue warp of both CTAs
    mbar_init(smem_u32(&bar_drain[0]), 1);
    mbar_init(smem_u32(&bar_drain[1]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                 "r"(static_cast<uint32_t>(C::kTmemCols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anything signals across the pair
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  pdl_wait();
  launder(slots);

  const int n_clusters = static_cast<int>(gridDim.x >> 1), cluster = static_cast<int>(blockIdx.x >> 1);
  const int total = (n_blocks + 1) / 2 * C::kTilePairs;

  // The issuing warpgroup and the two epilogue warpgroups do not meet again before the kernel's last lines.
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 0) {
      // ---------------------------------------------------------------- code producer (both CTAs)
      if (lane == 0) {
        const uint32_t full0 = map_to_cta(smem_u32(&bar_full[0]), 0);  // the leader's barriers, as seen from this CTA
        uint32_t it = 0, s = 0, ph = 1u;
        bool ok = true;
        for (int u = cluster; u < total && ok; u += n_clusters) {
          const int b = u / C::kTilePairs * 2 + static_cast<int>(rank), tp = u % C::kTilePairs;
          // the weights seen as rows of 128 bytes: a record is 128 rows of codes, 4 of scales, 4 of padding
          const int rec = (2 * tp + static_cast<int>(rank)) * C::kTilesK * 136;
          for (int kt = 0; kt < C::kTilesK; ++kt, ++it) {
            if (!mbar_wait(smem_u32(&bar_empty[s]), ph, abort_v, status)) { ok = false; break; }
            const uint32_t full = full0 + 8u * s, base = tiles + s * C::kStageBytes;
            if (leader) mbar_arrive_expect_tx(smem_u32(&bar_full[s]), 2 * C::kStageBytes);
            // token rows beyond the last (an odd block count, the ragged end) are read as zeros and count all the same
            tma_load_2d_pair(base + C::kTokOff, &map_x, kt * 128, b * 128, full);
            tma_load_2d_pair(base + C::kWOff, &map_wc, 0, rec + kt * 136, full);
            if (++s == C::kStages) { s = 0; ph ^= 1u; }
          }
        }
        if (!ok && leader) drain_copies(bar_full, it, C::kStages);
      }
    } else if (warp == 3) {
      // ---------------------------------------------------------------- scale producer (both CTAs)
      if (lane == 0) {
        const uint32_t sfull0 = map_to_cta(smem_u32(&bar_sfull[0]), 0);
        uint32_t it = 0;
        bool ok = true;
        for (int u = cluster; u < total && ok; u += n_clusters) {
          const int b = u / C::kTilePairs * 2 + static_cast<int>(rank), tp = u % C::kTilePairs;
          const int rec_lo = 2 * tp * C::kTilesK * 136 + 128, rec_hi = rec_lo + C::kTilesK * 136;
          for (int kt = 0; kt < C::kTilesK; ++kt, ++it) {
            const uint32_t j = it % C::kSfStages, ph = (it / C::kSfStages) & 1u;
            // free once its previous contents are in tensor memory
            if (!mbar_wait(smem_u32(&bar_sf[j]), ph ^ 1u, abort_v, status)) { ok = false; break; }
            const uint32_t sfull = sfull0 + 8u * j, slot = sf_ring + j * C::kSfSlotBytes;
            if (leader) mbar_arrive_expect_tx(smem_u32(&bar_sfull[j]), 2 * C::kSfSlotBytes);
            tma_load_2d_pair(slot + C::kSfTokOff, &map_sfx, 0, (b * C::kTilesK + kt) * 4, sfull);
            tma_load_2d_pair(slot + C::kSfWLoOff, &map_ws, 0, rec_lo + kt * 136, sfull);
            tma_load_2d_pair(slot + C::kSfWHiOff, &map_ws, 0, rec_hi + kt * 136, sfull);
          }
        }
        if (!ok && leader) drain_copies(bar_sfull, it, C::kSfStages);
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issue (leader only)
      if (leader) {
        // E4M3 x E4M3, UE8M0 scales, M = 256, N = 256; scale byte k of a row's cell for MMA k
        constexpr uint32_t kIdesc = (static_cast<uint32_t>(256 >> 3) << 17) | (1u << 23) | (static_cast<uint32_t>(256 >> 4) << 24);
        uint32_t ui = 0, s = 0, ph = 0, j = 0, sph = 0;
        bool ok = true, sf_ready = false, full_ready = false;
        for (int u = cluster; u < total && ok; u += n_clusters, ++ui) {
          if (!warp_wait(smem_u32(&bar_tempty), (ui & 1u) ^ 1u, abort_v, status)) break;
          tc_fence_after();
          for (int kt = 0; kt < C::kTilesK; ++kt) {
            if (!__all_sync(0xffffffffu, (sf_ready || mbar_wait(smem_u32(&bar_sf[j]), sph, abort_v, status)) &&
                                             (full_ready || mbar_wait(smem_u32(&bar_full[s]), ph, abort_v, status)))) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t s_now = s, j_now = j;
            if (++s == C::kStages) { s = 0; ph ^= 1u; }
            if (++j == C::kSfStages) { j = 0; sph ^= 1u; }
            sf_ready = mbar_test(smem_u32(&bar_sf[j]), sph);
            full_ready = mbar_test(smem_u32(&bar_full[s]), ph);
            const uint32_t lo = (tiles + s_now * C::kStageBytes) >> 4;
            const uint32_t x_lo = lo + (C::kTokOff >> 4), w_lo = lo + (C::kWOff >> 4);
            const uint32_t t_sft = tmem_base + C::kSfCol + 16u * j_now, t_sfw = t_sft + 8u;
            if (elect_one()) {
              tc_mma_mxf8_pair(tmem_base, x_lo, w_lo, kIdesc, t_sft, t_sfw, static_cast<uint32_t>(kt != 0));
              tc_mma_mxf8_pair(tmem_base, x_lo + 2, w_lo + 2, kIdesc | (1u << 29) | (1u << 4), t_sft, t_sfw, 1u);
              tc_mma_mxf8_pair(tmem_base, x_lo + 4, w_lo + 4, kIdesc | (2u << 29) | (2u << 4), t_sft, t_sfw, 1u);
              tc_mma_mxf8_pair(tmem_base, x_lo + 6, w_lo + 6, kIdesc | (3u << 29) | (3u << 4), t_sft, t_sfw, 1u);
              tc_commit_both(smem_u32(&bar_empty[s_now]));  // the stage is free again, in both CTAs
            }
            __syncwarp();
          }
          if (ok && elect_one()) tc_commit_both(smem_u32(&bar_tfull));
        }
        if (__any_sync(0xffffffffu, *abort_v != 0) && elect_one()) drain_tcgen05_pair(smem_u32(&bar_drain[0]));
      }
    } else {
      // ---------------------------------------------------------------- scale copies into both CTAs' tensor memory (leader)
      if (leader) {
        uint32_t s = 0, ph = 1u, j = 0, sph = 0;
        bool ok = true, landed = false, free_set = false;
        for (int u = cluster; u < total && ok; u += n_clusters) {
          for (int kt = 0; kt < C::kTilesK; ++kt) {
            // set j was last read by the MMAs 8 K-tiles back: complete once those that read stage s, kStages back, are
            if (!__all_sync(0xffffffffu, (landed || mbar_wait(smem_u32(&bar_sfull[j]), sph, abort_v, status)) &&
                                             (free_set || mbar_wait(smem_u32(&bar_empty[s]), ph, abort_v, status)))) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t lo = (sf_ring + j * C::kSfSlotBytes) >> 4, sf_bar = smem_u32(&bar_sf[j]);
            const uint32_t t_sft = tmem_base + C::kSfCol + 16u * j, t_sfw = t_sft + 8u;
            if (++s == C::kStages) { s = 0; ph ^= 1u; }
            if (++j == C::kSfStages) { j = 0; sph ^= 1u; }
            landed = mbar_test(smem_u32(&bar_sfull[j]), sph);
            free_set = mbar_test(smem_u32(&bar_empty[s]), ph);
            if (elect_one()) {
              tc_cp_scales_pair(t_sft, lo + (C::kSfTokOff >> 4));      // each CTA its own token rows
              tc_cp_scales_pair(t_sfw, lo + (C::kSfWLoOff >> 4));      // weight rows 0..127 of N
              tc_cp_scales_pair(t_sfw + 4, lo + (C::kSfWHiOff >> 4));  // 128..255
              tc_commit_both(sf_bar);
            }
            __syncwarp();
          }
        }
        if (__any_sync(0xffffffffu, *abort_v != 0) && elect_one()) drain_tcgen05_pair(smem_u32(&bar_drain[1]));
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue (both CTAs, warps 4..11)
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    const int q = warp & 3;                  // the TMEM lane quarter this warp may read
    const int half = (warp >> 2) - 1;        // which weight tile of the pair
    const int tr = q * 32 + lane;            // token row inside the block = TMEM lane
    const uint32_t tempty_leader = map_to_cta(smem_u32(&bar_tempty), 0);
    uint8_t* strip = smem_raw + (tiles - smem_u32(smem_raw)) + C::kStripOff + (warp - 4) * C::kStripBytes;
    uint32_t ui = 0;
    const int lane_row = lane / C::kLanesPerRow, lane_col = (lane & (C::kLanesPerRow - 1)) * 8;
    // MODE 3: the slots of part `part` (rows 8 * part ..) of unit v, four rows per lane
    const auto load_slots = [&](int v, int part, uint4 (&s)[4][4]) {
      const int64_t r0 = static_cast<int64_t>(v / C::kTilePairs * 2 + static_cast<int>(rank)) * 128 + q * 32 + C::kPartRows * part;
      const __nv_bfloat16* src = slots + (2 * (v % C::kTilePairs) + half) * 128 + lane_col;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int64_t r = r0 + 32 / C::kLanesPerRow * i + lane_row;
#pragma unroll
        for (int k = 0; k < kTopK; ++k)
          s[i][k] = v < total && r < tokens ? __ldcg(reinterpret_cast<const uint4*>(src + (r * kTopK + k) * kH)) : uint4{};
      }
    };
    uint4 ahead[MODE == 3 ? 2 : 1][4][4];
    if (MODE == 3) load_slots(cluster, 0, ahead[0]);
    for (int u = cluster; u < total; u += n_clusters, ++ui) {
      const int b = u / C::kTilePairs * 2 + static_cast<int>(rank), tp = u % C::kTilePairs;
      const bool have_rows = b < n_blocks;
      const int64_t row = static_cast<int64_t>(b) * 128 + tr;
      // the warp decides together: tcgen05.ld below needs all 32 lanes
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_tfull), ui & 1u, abort_v, status))) break;
      tc_fence_after();
      const uint32_t t_acc = tmem_base + 128u * half + (static_cast<uint32_t>(q * 32) << 16);
      uint32_t acc[MODE == 1 ? 4 : 2][32];
      uint4 packed[MODE == 1 ? 1 : 2][8];  // MODE 2, 3: the row's 128 values in bf16
      if (have_rows && MODE == 1) {
        tc_ld32_nowait(t_acc, acc[0]);
        tc_ld32_nowait(t_acc + 32, acc[1]);
        tc_ld32_nowait(t_acc + 64, acc[MODE == 1 ? 2 : 0]);
        tc_ld32_nowait(t_acc + 96, acc[MODE == 1 ? 3 : 0]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      } else if (have_rows) {
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          tc_ld32_nowait(t_acc + 64 * hh, acc[0]);
          tc_ld32_nowait(t_acc + 64 * hh + 32, acc[1]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            uint32_t o[4];
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
              const int c = 8 * (k & 3) + 2 * jj;
              const __nv_bfloat162 p2 = __floats2bfloat162_rn(__uint_as_float(acc[k >> 2][c]), __uint_as_float(acc[k >> 2][c + 1]));
              o[jj] = *reinterpret_cast<const uint32_t*>(&p2);
            }
            packed[MODE == 1 ? 0 : hh][k] = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(tempty_leader);
      if (!have_rows) {
        if (MODE == 3) load_slots(u + n_clusters, 0, ahead[0]);
        continue;
      }
      if (MODE == 1) {
        // columns of a tile: [gate 32 | up 32 | gate 32 | up 32] of 64 intermediate columns
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          float h[32];
          float amax = 0.0f;
#pragma unroll
          for (int k = 0; k < 32; ++k) {
            h[k] = swiglu_oai(__uint_as_float(acc[MODE == 1 ? 2 * g : 0][k]), __uint_as_float(acc[MODE == 1 ? 2 * g + 1 : 0][k]));
            amax = fmaxf(amax, fabsf(h[k]));
          }
          const int sc = mxfp8_scale(amax);
          const float inv = __uint_as_float(static_cast<uint32_t>(254 - sc) << 23);
          uint32_t words[8];
#pragma unroll
          for (int wd = 0; wd < 8; ++wd)
            words[wd] = cvt_e4m3x2(h[4 * wd] * inv, h[4 * wd + 1] * inv) |
                        (cvt_e4m3x2(h[4 * wd + 2] * inv, h[4 * wd + 3] * inv) << 16);
          const int grp = 4 * tp + 2 * half + g;
          uint4* dst = reinterpret_cast<uint4*>(h8 + row * kI + grp * 32);
          dst[0] = make_uint4(words[0], words[1], words[2], words[3]);
          dst[1] = make_uint4(words[4], words[5], words[6], words[7]);
          sfh8[(static_cast<int64_t>(b) * kS2TilesK + (grp >> 2)) * kAtomBytes + atom_offset(tr, grp & 3)] =
              static_cast<uint8_t>(sc);
        }
      } else {
        const int64_t row0 = static_cast<int64_t>(b) * 128 + q * 32;
        __nv_bfloat16* dst0 = out + row0 * kH + (2 * tp + half) * 128 + lane_col;
        constexpr int kRowParts = 32 / C::kPartRows;
#pragma unroll
        for (int part = 0; part < 4; ++part) {
          const int hh = part / kRowParts, p = part % kRowParts;  // columns, rows
          if (MODE == 3) load_slots(part < 3 ? u : u + n_clusters, (part + 1) & 3, ahead[(part + 1) & (MODE == 3)]);
          if (lane / C::kPartRows == p) {
#pragma unroll
            for (int k = 0; k < C::kLanesPerRow; ++k) {
              const int chunk = hh * C::kLanesPerRow + k;
              *reinterpret_cast<uint4*>(strip + (lane & (C::kPartRows - 1)) * C::kStripRow + k * 16) =
                  packed[MODE == 1 ? 0 : chunk >> 3][chunk & 7];
            }
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = 32 / C::kLanesPerRow * i + lane_row;
            uint4 val = *reinterpret_cast<const uint4*>(strip + r * C::kStripRow + lane_col * 2);
            if (MODE == 3) {
              float sum[8] = {};
#pragma unroll
              for (int k = 0; k < kTopK; ++k) add_bf16x8(sum, ahead[part & (MODE == 3)][i][k]);
              add_bf16x8(sum, val);
              uint32_t o[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const __nv_bfloat162 p2 = __floats2bfloat162_rn(sum[2 * k], sum[2 * k + 1]);
                o[k] = *reinterpret_cast<const uint32_t*>(&p2);
              }
              val = make_uint4(o[0], o[1], o[2], o[3]);
            }
            if (row0 + C::kPartRows * p + r < tokens)
              *reinterpret_cast<uint4*>(dst0 + static_cast<int64_t>(C::kPartRows * p + r) * kH + hh * 64) = val;
          }
          __syncwarp();
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA frees tensor memory or leaves while the partner may still signal or read it
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(C::kTmemCols))
                 : "memory");
  }
}

// ------------------------------------------------------------------------------------------------ host side
template <int MODE>
static int shared_pairs() {
  static std::mutex mu;
  static int pairs[kMaxDevices] = {};
  static bool known[kMaxDevices] = {};
  return resident_pairs_of(shared_pair_kernel<MODE>, SharedPairCfg<MODE>::kThreads, SharedPairCfg<MODE>::kSmemBytes, mu, known,
                           pairs);
}

template <int MODE>
static int launch_shared_pair(const CUtensorMap& mx, const uint8_t* w_tiles, const uint8_t* sf_x, const SharedWorkspace& ws,
                              int64_t tokens, const void* slots_bf16, void* out_bf16, int32_t* status, cudaStream_t stream) {
  using C = SharedPairCfg<MODE>;
  CUtensorMap msf, mwc, mws;
  const int n_blocks = static_cast<int>(ws.rows / 128);
  const uint64_t w_rows = static_cast<uint64_t>(C::kTilesM) * C::kTilesK * 136;
  int r;
  if ((r = make_flat_map(&msf, sf_x, static_cast<uint64_t>(n_blocks) * C::kTilesK * 4, 4))) return r;
  if ((r = make_flat_map(&mwc, w_tiles, w_rows, 128))) return r;
  if ((r = make_flat_map(&mws, w_tiles, w_rows, 4))) return r;
  const int units = (n_blocks + 1) / 2 * C::kTilePairs, pairs = shared_pairs<MODE>();
  return launch_pairs(shared_pair_kernel<MODE>, units < pairs ? units : pairs, C::kThreads, C::kSmemBytes, stream, mx, msf, mwc,
                      mws, n_blocks, tokens, ws.h8, ws.sfh8, static_cast<const __nv_bfloat16*>(slots_bf16),
                      static_cast<__nv_bfloat16*>(out_bf16), status);
}

bool shared_pair_supported() { return shared_pairs<1>() > 0 && shared_pairs<2>() > 0 && shared_pairs<3>() > 0; }

// The GEMMs on blocks of 128 tokens (ws.bm == 128). `map_x` / `map_h`: the token codes and h as 128-byte swizzled boxes of 128.
int shared_pair_gemm1(const CUtensorMap& map_x, const uint8_t* w13t, const SharedWorkspace& ws, int64_t tokens, int32_t* status,
                      cudaStream_t stream) {
  return launch_shared_pair<1>(map_x, w13t, ws.sfx8, ws, tokens, nullptr, nullptr, status, stream);
}
// slots_bf16 null: the shared rows; else the sum of the four slots and the shared row
int shared_pair_gemm2(const CUtensorMap& map_h, const uint8_t* w2t, const SharedWorkspace& ws, const void* slots_bf16,
                      void* out_bf16, int64_t tokens, int32_t* status, cudaStream_t stream) {
  return slots_bf16 ? launch_shared_pair<3>(map_h, w2t, ws.sfh8, ws, tokens, slots_bf16, out_bf16, status, stream)
                    : launch_shared_pair<2>(map_h, w2t, ws.sfh8, ws, tokens, nullptr, out_bf16, status, stream);
}

int set_wait_limit_shared_pair(unsigned long long ns) { return set_wait_limit_here(ns); }

}  // namespace b200moe
