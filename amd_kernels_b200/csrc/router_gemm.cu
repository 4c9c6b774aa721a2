// Router GEMM on the CUDA cores: bf16 activations x fp32 gate -> fp32 split-K partial logits [S][T][E], consumed by the
// top-4 kernel, which adds the partials from 0.0 in split order. Products are exact in fp32 (a bf16 factor has 8 significant
// bits) and each partial is short fp32 FMA chains joined by a tree, so the error per partial stays far below
// 2^-18 * sum|x||w| (the bound the reference states for its three-term bf16 split).
//
// A partial is ONE chain of FMAs over the K elements of its split, in rising K from 0.0: the sum does not depend on the
// token count or on how the work is dealt, and a change of tiling here never moves a logit's last bit.
//
// Used below 128 tokens, where the product is latency: 3.1 MB of gate, 12 KB of x per token. A CTA owns 16 experts x one K
// split x 16 tokens, so one token alone already spreads the gate over 128 CTAs (with 16 splits) of 24 KB each, fetched in one
// batch of asynchronous copies. Measured with both quantisers, us back to back: 4.0 / 9.9 / 10.4 / 10.6 / 18.8 at 1 / 16 / 32 /
// 64 / 100 tokens. K dealt over the lanes of a warp and joined by a tree takes 3.9 / 3.9 / 4.5 / 8.7 / 13.8, but its sums
// have other last bits, which reach the weights and through them the layer's result.
#include "common.cuh"

namespace b200moe {

constexpr int kRgTokens = 16;             // tokens per CTA
constexpr int kRgExperts = 16;            // experts per CTA
constexpr int kRgChunk = 384;             // K elements in shared memory at a time
constexpr int kRgVecs = kRgChunk / 4;     // 16-byte vectors of a row of them
constexpr int kRgPerThread = 2;           // tokens (chains) per thread
constexpr int kRgThreads = kRgTokens * kRgExperts / kRgPerThread;

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

// 16 bytes from an address that need not be aligned (`vec`: it is)
__device__ __forceinline__ uint4 load_bf16x8(const __nv_bfloat16* p, bool vec) {
  if (vec) return __ldcg(reinterpret_cast<const uint4*>(p));
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

// vector c of row r in shared memory: the eight lanes of a load phase read one c of eight rows, so the vectors of a row are
// permuted by the row to spread those over the banks
__device__ __forceinline__ int rg_at(int r, int c) { return r * kRgVecs + (c ^ (r & 7)); }

// grid (ceil(E / 16), S, ceil(T / 16)); thread: one expert (tid % 16), the tokens tid / 16 and tid / 16 + 8 of the CTA's
template <bool QUANT>
__global__ void __launch_bounds__(kRgThreads) router_gemm_kernel(const __nv_bfloat16* __restrict__ x,
                                                                 const float* __restrict__ gate, int64_t tokens,
                                                                 int num_experts, int k_per_split,
                                                                 float* __restrict__ partials, QuantOut q, bool vec) {
  __shared__ float4 ws[kRgExperts * kRgVecs];
  __shared__ float4 xs[kRgTokens * kRgVecs];
  const int tid = threadIdx.x;
  const int e0 = blockIdx.x * kRgExperts, e = tid % kRgExperts, tg = tid / kRgExperts;
  constexpr int kGroups = kRgThreads / kRgExperts;
  const int64_t t0 = static_cast<int64_t>(blockIdx.z) * kRgTokens;
  const int nt = static_cast<int>(min(static_cast<int64_t>(kRgTokens), tokens - t0));
  const int k0 = blockIdx.y * k_per_split;
  // this CTA's slice of the gate: into L2 before the wait, read behind it (the work in front may have written it)
  if (vec && tid < kRgExperts && e0 + tid < num_experts)
    l2_prefetch_bulk(gate + static_cast<int64_t>(e0 + tid) * kH + k0, static_cast<uint32_t>(k_per_split * 4));
  pdl_enter(x, gate);
  auto load_gate = [&](int kk) {
    const int vecs = min(kRgChunk, k_per_split - kk) / 4;
    for (int i = tid; i < kRgExperts * kRgVecs; i += kRgThreads) {
      const int r = i / kRgVecs, c = i % kRgVecs;
      if (c >= vecs || e0 + r >= num_experts) continue;  // never read
      const float* src = gate + static_cast<int64_t>(e0 + r) * kH + k0 + kk + 4 * c;
      float4* dst = ws + rg_at(r, c);
      if (vec)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                     "l"(src)
                     : "memory");
      else
        *dst = make_float4(__ldcg(src), __ldcg(src + 1), __ldcg(src + 2), __ldcg(src + 3));
    }
  };
  load_gate(0);
  float acc[kRgPerThread];
  int row[kRgPerThread];  // (rows beyond the last token: the last one again, not stored)
#pragma unroll
  for (int j = 0; j < kRgPerThread; ++j) {
    acc[j] = 0.0f;
    row[j] = min(tg + j * kGroups, nt - 1);
  }
  for (int kk = 0; kk < k_per_split; kk += kRgChunk) {
    const int chunk = min(kRgChunk, k_per_split - kk), v8s = chunk / 8;  // 16-byte vectors of a bf16 row in this chunk
    if (kk) {
      __syncthreads();
      load_gate(kk);
    }
    for (int i = tid; i < nt * v8s; i += kRgThreads) {
      const int r = i / v8s, c = i % v8s;
      const uint4 raw = load_bf16x8(x + (t0 + r) * kH + k0 + kk + 8 * c, vec);
      xs[rg_at(r, 2 * c)] = make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u),
                                        __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
      xs[rg_at(r, 2 * c + 1)] = make_float4(__uint_as_float(raw.z << 16), __uint_as_float(raw.z & 0xffff0000u),
                                            __uint_as_float(raw.w << 16), __uint_as_float(raw.w & 0xffff0000u));
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (QUANT) {
      // one pass over x: the CTAs of the expert groups share the chunk's blocks of 32 values; 4 threads x 8 values per block
      const int groups = gridDim.x, mine = (nt - static_cast<int>(blockIdx.x) + groups - 1) / groups;  // tokens of this CTA
      for (int i = tid; i < ((mine * v8s + 31) & ~31); i += kRgThreads) {  // whole warps stay together for the shuffles
        const bool live = i < mine * v8s;
        const int r = live ? (i / v8s) * groups + static_cast<int>(blockIdx.x) : 0, v8 = live ? i % v8s : 0;
        const float4 lo = xs[rg_at(r, 2 * v8)], hi = xs[rg_at(r, 2 * v8 + 1)];
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
#pragma unroll 8
      for (int c = 0; c < chunk / 4; ++c) {
        const float4 w = ws[rg_at(e, c)];
#pragma unroll
        for (int j = 0; j < kRgPerThread; ++j) {
          const float4 v = xs[rg_at(row[j], c)];
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
  for (int j = 0; j < kRgPerThread; ++j)
    if (tg + j * kGroups < nt)
      partials[(static_cast<int64_t>(blockIdx.y) * tokens + t0 + tg + j * kGroups) * num_experts + e0 + e] = acc[j];
}

static bool aligned16(const void* a, const void* b, const void* c, const void* d) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
           reinterpret_cast<uintptr_t>(d)) & 15) == 0;
}

}  // namespace b200moe

extern "C" int b200moe_router_splits(int64_t tokens) { return tokens <= 2048 ? 16 : 4; }

extern "C" int b200moe_router_gemm(const void* x_bf16, const float* gate, int64_t tokens, int num_experts, int splits,
                                   float* partials, void* stream) {
  using namespace b200moe;
  if (!x_bf16 || !gate || !partials || tokens < 0 || num_experts < 1 || num_experts > kMaxE) return B200MOE_E_ARG;
  if (splits < 1 || kH % splits || (kH / splits) % 32) return B200MOE_E_ARG;
  if (tokens == 0) return 0;
  const dim3 grid(static_cast<unsigned>((num_experts + kRgExperts - 1) / kRgExperts), static_cast<unsigned>(splits),
                  static_cast<unsigned>((tokens + kRgTokens - 1) / kRgTokens));
  B200MOE_LAUNCH(router_gemm_kernel<false>, grid, kRgThreads, 0, static_cast<cudaStream_t>(stream),
                 static_cast<const __nv_bfloat16*>(x_bf16), gate, tokens, num_experts, kH / splits, partials, QuantOut{},
                 aligned16(x_bf16, gate, nullptr, nullptr));
  return 0;
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
  const dim3 grid(static_cast<unsigned>((num_experts + kRgExperts - 1) / kRgExperts), static_cast<unsigned>(splits),
                  static_cast<unsigned>((tokens + kRgTokens - 1) / kRgTokens));
  const QuantOut q{codes4, scales4, codes8, scales8, atoms8, shift};
  B200MOE_LAUNCH(router_gemm_kernel<true>, grid, kRgThreads, 0, static_cast<cudaStream_t>(stream),
                 static_cast<const __nv_bfloat16*>(x_bf16), gate, tokens, num_experts, kH / splits, partials, q,
                 aligned16(x_bf16, gate, codes4, codes8));
  return 0;
}
}  // namespace b200moe

extern "C" int b200moe_router_gemm_quant(const void* x_bf16, const float* gate, int64_t tokens, int num_experts, int splits,
                                         float* partials, uint8_t* codes4, uint8_t* scales4, uint8_t* codes8,
                                         uint8_t* scales8, void* stream) {
  return b200moe::router_gemm_quant(x_bf16, gate, tokens, num_experts, splits, partials, codes4, scales4, codes8, scales8,
                                    nullptr, 16, stream);
}
