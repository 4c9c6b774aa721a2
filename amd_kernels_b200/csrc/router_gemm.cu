// Router GEMM on the CUDA cores: bf16 activations x fp32 gate -> fp32 split-K partial logits [S][T][E], consumed by the
// top-4 kernel, which adds the partials from 0.0 in split order. Products are exact in fp32 (a bf16 factor has 8 significant
// bits) and each partial is a short fp32 FMA chain, so the error per partial stays far below 2^-18 * sum|x||w| (the bound the
// reference states for its three-term bf16 split).
//
// A partial is ONE chain of FMAs over the K elements of its split, in rising K from 0.0: the sum does not depend on the
// token count or on how the work is dealt, and a change of tiling here never moves a logit's last bit.
//
// Used below 128 tokens, where the product is latency: 3.1 MB of gate, 12 KB of x per token. A CTA owns 16 experts x one K
// split x 16 (32) tokens, so one token alone already spreads the gate over 128 CTAs (with 16 splits) of 24 KB each, fetched in
// one batch of asynchronous copies. What bounds it is how fast a warp issues -- one instruction in three to five cycles with
// one warp per scheduler -- so eight warps with few instructions each: a thread runs one chain (two), both factors come from shared
// memory in 16-byte loads at constant offsets, and rows are padded so that the rows of a load lie on different banks.
// Measured with both quantisers, us back to back: 4.0 / 4.0 / 7.3 / 7.8 / 10.0 / 15.8 at 1 / 8 / 16 / 32 / 64 / 100 tokens. With
// four warps, rows permuted instead of padded and x fetched row by row it took 4.0 / 8.5 / 9.9 / 10.4 / 10.6 / 18.7; with the chain
// passed through 16 lanes and the gate in registers 10.8 / 13.2 / 15.9 / 21.7 / 22.6 / 22.9; with K dealt over the lanes and joined
// by a tree 3.9 / 3.9 / 3.9 / 4.5 / 8.7 / 13.8, but those sums have other last bits, which reach the layer's result.
#include "common.cuh"
#include "tc_host.cuh"

namespace b200moe {

constexpr int kRgExperts = 16;            // experts per CTA
constexpr int kRgChunk = 384;             // K elements in shared memory at a time
constexpr int kRgVecs = kRgChunk / 4;     // 16-byte vectors of a row of them
constexpr int kRgStride = kRgVecs + 1;    // of a row in shared memory: neighbouring rows start on other banks
constexpr int kRgThreads = 256;
constexpr int kRgGroups = kRgThreads / kRgExperts;
// tokens of a CTA: PT chains per thread
template <int PT>
constexpr int rg_smem() { return (kRgExperts + kRgGroups * PT) * kRgStride * 16; }

// What the fused form also writes, row-major: the routed experts' MXFP4 operands and (optionally) the shared expert's
// MXFP8 operands of the same rows.
struct QuantOut {
  uint8_t* codes4;   // [T][3072]
  uint8_t* scales4;  // [T][192]
  uint8_t* codes8;   // [T][6144], may be null
  uint8_t* scales8;  // [T][192], or null:
  uint8_t* atoms8;   // the same bytes as the scale atoms of 2^atom_shift-row blocks
  int atom_shift;
};

// 16 bytes from an address that is not aligned
__device__ __forceinline__ uint4 load_bf16x8(const __nv_bfloat16* p) {
  const unsigned short* h = reinterpret_cast<const unsigned short*>(p);
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) w[j] = static_cast<uint32_t>(__ldcg(h + 2 * j)) | (static_cast<uint32_t>(__ldcg(h + 2 * j + 1)) << 16);
  return make_uint4(w[0], w[1], w[2], w[3]);
}
template <typename T>
__device__ __forceinline__ void store_bytes(uint8_t* p, T v, bool vec) {
  if (vec) {
    *reinterpret_cast<T*>(p) = v;
  } else {
    for (int i = 0; i < static_cast<int>(sizeof(T)); ++i) p[i] = reinterpret_cast<const uint8_t*>(&v)[i];
  }
}

// grid (ceil(E / 16), S, ceil(T / (16 PT))); thread: one expert (tid % 16), the tokens tid / 16 + 16 j of the CTA's
template <bool QUANT, int PT>
__global__ void __launch_bounds__(kRgThreads) router_gemm_kernel(const __nv_bfloat16* __restrict__ x,
                                                                 const float* __restrict__ gate, int64_t tokens,
                                                                 int num_experts, int k_per_split,
                                                                 float* __restrict__ partials, QuantOut q, bool vec) {
  constexpr int kTokens = kRgGroups * PT;
  extern __shared__ float4 rg_smem_raw[];
  float4(*ws)[kRgStride] = reinterpret_cast<float4(*)[kRgStride]>(rg_smem_raw);
  float4(*xs)[kRgStride] = ws + kRgExperts;
  const int tid = threadIdx.x;
  const int e0 = blockIdx.x * kRgExperts, e = tid % kRgExperts, tg = tid / kRgExperts;
  const int64_t t0 = static_cast<int64_t>(blockIdx.z) * kTokens;
  const int nt = static_cast<int>(min(static_cast<int64_t>(kTokens), tokens - t0));
  const int k0 = blockIdx.y * k_per_split;
  // this CTA's slice of the gate: into L2 before the wait, read behind it (the work in front may have written it)
  if (vec && tid < kRgExperts && e0 + tid < num_experts)
    l2_prefetch_bulk(gate + static_cast<int64_t>(e0 + tid) * kH + k0, static_cast<uint32_t>(k_per_split * 4));
  pdl_enter(x, gate);
  auto load_gate = [&](int kk) {
    const int vecs = min(kRgChunk, k_per_split - kk) / 4;
#pragma unroll
    for (int it = 0; it < kRgExperts * kRgVecs / kRgThreads; ++it) {
      const int i = it * kRgThreads + tid, r = i / kRgVecs, c = i % kRgVecs;
      if (c >= vecs || e0 + r >= num_experts) continue;  // never read
      const float* src = gate + static_cast<int64_t>(e0 + r) * kH + k0 + kk + 4 * c;
      float4* dst = &ws[r][c];
      if (vec)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                     "l"(src)
                     : "memory");
      else
        *dst = make_float4(__ldcg(src), __ldcg(src + 1), __ldcg(src + 2), __ldcg(src + 3));
    }
  };
  load_gate(0);
  float acc[PT];
  const float4* row[PT];  // (rows beyond the last token: the last one again, not stored)
#pragma unroll
  for (int j = 0; j < PT; ++j) {
    acc[j] = 0.0f;
    row[j] = xs[min(tg + j * kRgGroups, nt - 1)];
  }
  for (int kk = 0; kk < k_per_split; kk += kRgChunk) {
    const int chunk = min(kRgChunk, k_per_split - kk), v8s = chunk / 8;  // 16-byte vectors of a bf16 row in this chunk
    if (kk) {
      __syncthreads();
      load_gate(kk);
    }
    constexpr int kLoads = kTokens * kRgChunk / 8 / kRgThreads;  // of a thread, all in flight together
    uint4 raw[kLoads];
    if (vec) {
#pragma unroll
      for (int it = 0; it < kLoads; ++it) {
        const int i = it * kRgThreads + tid, r = i / (kRgChunk / 8), c = i % (kRgChunk / 8);
        if (r < nt && c < v8s) raw[it] = __ldcg(reinterpret_cast<const uint4*>(x + (t0 + r) * kH + k0 + kk + 8 * c));
      }
    } else {
#pragma unroll
      for (int it = 0; it < kLoads; ++it) {
        const int i = it * kRgThreads + tid, r = i / (kRgChunk / 8), c = i % (kRgChunk / 8);
        if (r < nt && c < v8s) raw[it] = load_bf16x8(x + (t0 + r) * kH + k0 + kk + 8 * c);
      }
    }
#pragma unroll
    for (int it = 0; it < kLoads; ++it) {
      const int i = it * kRgThreads + tid, r = i / (kRgChunk / 8), c = i % (kRgChunk / 8);
      if (r < nt && c < v8s) {
        xs[r][2 * c] = make_float4(__uint_as_float(raw[it].x << 16), __uint_as_float(raw[it].x & 0xffff0000u),
                                   __uint_as_float(raw[it].y << 16), __uint_as_float(raw[it].y & 0xffff0000u));
        xs[r][2 * c + 1] = make_float4(__uint_as_float(raw[it].z << 16), __uint_as_float(raw[it].z & 0xffff0000u),
                                       __uint_as_float(raw[it].w << 16), __uint_as_float(raw[it].w & 0xffff0000u));
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (QUANT) {
      // one pass over x: the CTAs of the expert groups share the chunk's blocks of 32 values; 4 threads x 8 values per block
      const int groups = gridDim.x, mine = (nt - static_cast<int>(blockIdx.x) + groups - 1) / groups;  // tokens of this CTA
      for (int i = tid; i < ((mine * v8s + 31) & ~31); i += kRgThreads) {  // whole warps stay together for the shuffles
        const bool live = i < mine * v8s;
        const int r = live ? (i / v8s) * groups + static_cast<int>(blockIdx.x) : 0, v8 = live ? i % v8s : 0;
        const float4 lo = xs[r][2 * v8], hi = xs[r][2 * v8 + 1];
        const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        float amax = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        if (!live) continue;
        const int64_t t = t0 + r;
        const int k = k0 + kk + 8 * v8;
        const int e4 = quark_even_e8m0(amax);
        const float inv4 = __uint_as_float(static_cast<uint32_t>(254 - e4) << 23);
        uint32_t packed = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) packed |= cvt_e2m1x2(v[2 * j] * inv4, v[2 * j + 1] * inv4) << (8 * j);
        store_bytes(q.codes4 + t * (kH / 2) + (k >> 1), packed, vec);
        if ((v8 & 3) == 0) q.scales4[t * (kH / 32) + (k >> 5)] = static_cast<uint8_t>(e4);
        if (q.codes8 != nullptr) {
          const int e8 = mxfp8_scale(amax);
          const float inv8 = __uint_as_float(static_cast<uint32_t>(254 - e8) << 23);
          store_bytes(q.codes8 + t * kH + k,
              make_uint2(cvt_e4m3x2(v[0] * inv8, v[1] * inv8) | (cvt_e4m3x2(v[2] * inv8, v[3] * inv8) << 16),
                         cvt_e4m3x2(v[4] * inv8, v[5] * inv8) | (cvt_e4m3x2(v[6] * inv8, v[7] * inv8) << 16)), vec);
          if ((v8 & 3) == 0) {
            uint8_t* dst = q.scales8 != nullptr
                               ? q.scales8 + t * (kH / 32) + (k >> 5)
                               : q.atoms8 + ((t >> q.atom_shift) * (kH / 128) + (k >> 7)) * kAtomBytes +
                                     atom_offset(static_cast<int>(t & ((1 << q.atom_shift) - 1)), (k >> 5) & 3);
            *dst = static_cast<uint8_t>(e8);
          }
        }
      }
    }
    if (tg < nt) {
#pragma unroll 16
      for (int c = 0; c < chunk / 4; ++c) {
        const float4 w = ws[e][c];
#pragma unroll
        for (int j = 0; j < PT; ++j) {
          const float4 v = row[j][c];
          acc[j] = fmaf(v.x, w.x, acc[j]);
          acc[j] = fmaf(v.y, w.y, acc[j]);
          acc[j] = fmaf(v.z, w.z, acc[j]);
          acc[j] = fmaf(v.w, w.w, acc[j]);
        }
      }
    }
  }
  if (e0 + e >= num_experts) return;
#pragma unroll
  for (int j = 0; j < PT; ++j)
    if (tg + j * kRgGroups < nt)
      partials[(static_cast<int64_t>(blockIdx.y) * tokens + t0 + tg + j * kRgGroups) * num_experts + e0 + e] = acc[j];
}

static bool aligned16(const void* a, const void* b, const void* c, const void* d) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
           reinterpret_cast<uintptr_t>(d)) & 15) == 0;
}

template <bool QUANT, int PT>
static int launch_router(const void* x, const float* gate, int64_t tokens, int num_experts, int splits, float* partials,
                         const QuantOut& q, bool vec, cudaStream_t stream) {
  static PerDeviceOnce once;
  const int rc = once.run([] {
    return static_cast<int>(cudaFuncSetAttribute(router_gemm_kernel<QUANT, PT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 rg_smem<PT>()));
  });
  if (rc) return rc;
  constexpr int kTokens = kRgGroups * PT;
  const dim3 grid(static_cast<unsigned>((num_experts + kRgExperts - 1) / kRgExperts), static_cast<unsigned>(splits),
                  static_cast<unsigned>((tokens + kTokens - 1) / kTokens));
  B200MOE_LAUNCH((router_gemm_kernel<QUANT, PT>), grid, kRgThreads, rg_smem<PT>(), stream, static_cast<const __nv_bfloat16*>(x),
                 gate, tokens, num_experts, kH / splits, partials, q, vec);
  return 0;
}
// Up to 32 tokens one chain per thread: the time is a chain's latency (7.8 us at 32 tokens, 9.7 with two). Above, two: half the
// gate traffic and fewer loads per FMA (10.0 us at 64 tokens and 15.8 at 100, 14.1 and 21.3 with one).
constexpr int64_t kRgOneChain = 32;
template <bool QUANT>
static int launch_router_any(const void* x, const float* gate, int64_t tokens, int num_experts, int splits, float* partials,
                             const QuantOut& q, bool vec, cudaStream_t stream) {
  return tokens <= kRgOneChain ? launch_router<QUANT, 1>(x, gate, tokens, num_experts, splits, partials, q, vec, stream)
                               : launch_router<QUANT, 2>(x, gate, tokens, num_experts, splits, partials, q, vec, stream);
}

}  // namespace b200moe

extern "C" int b200moe_router_splits(int64_t tokens) { return tokens <= 2048 ? 16 : 4; }

extern "C" int b200moe_router_gemm(const void* x_bf16, const float* gate, int64_t tokens, int num_experts, int splits,
                                   float* partials, void* stream) {
  using namespace b200moe;
  if (!x_bf16 || !gate || !partials || tokens < 0 || num_experts < 1 || num_experts > kMaxE) return B200MOE_E_ARG;
  if (splits < 1 || kH % splits || (kH / splits) % 32) return B200MOE_E_ARG;
  if (tokens == 0) return 0;
  return launch_router_any<false>(x_bf16, gate, tokens, num_experts, splits, partials, QuantOut{},
                                  aligned16(x_bf16, gate, nullptr, nullptr), static_cast<cudaStream_t>(stream));
}

namespace b200moe {
// b200moe_router_gemm_quant; the shared expert's scales as rows (scales8) or as the atoms of bm8-row blocks (atoms8)
int router_gemm_quant(const void* x_bf16, const float* gate, int64_t tokens, int num_experts, int splits, float* partials,
                      uint8_t* codes4, uint8_t* scales4, uint8_t* codes8, uint8_t* scales8, uint8_t* atoms8, int bm8,
                      void* stream) {
  if (!x_bf16 || !gate || !partials || !codes4 || !scales4 || tokens < 0 || num_experts < 1 || num_experts > kMaxE)
    return B200MOE_E_ARG;
  if ((codes8 != nullptr) != (scales8 != nullptr || atoms8 != nullptr)) return B200MOE_E_ARG;
  if (splits < 1 || kH % splits || (kH / splits) % 32) return B200MOE_E_ARG;
  if (reinterpret_cast<uintptr_t>(codes8) & 1) return B200MOE_E_ALIGN;
  if (tokens == 0) return 0;
  const int shift = bm8 == 16 ? 4 : bm8 == 32 ? 5 : bm8 == 64 ? 6 : 7;
  return launch_router_any<true>(x_bf16, gate, tokens, num_experts, splits, partials,
                                 QuantOut{codes4, scales4, codes8, scales8, atoms8, shift}, aligned16(x_bf16, gate, codes4, codes8),
                                 static_cast<cudaStream_t>(stream));
}
}  // namespace b200moe

extern "C" int b200moe_router_gemm_quant(const void* x_bf16, const float* gate, int64_t tokens, int num_experts, int splits,
                                         float* partials, uint8_t* codes4, uint8_t* scales4, uint8_t* codes8,
                                         uint8_t* scales8, void* stream) {
  return b200moe::router_gemm_quant(x_bf16, gate, tokens, num_experts, splits, partials, codes4, scales4, codes8, scales8,
                                    nullptr, 16, stream);
}
