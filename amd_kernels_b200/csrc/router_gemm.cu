// Router GEMM on the CUDA cores: bf16 activations x fp32 gate -> fp32 split-K partial logits [S][T][E], consumed by the
// top-4 kernel, which adds the partials from 0.0 in split order. Products are exact in fp32 (a bf16 factor has 8 significant
// bits) and each partial is short fp32 FMA chains joined by a tree, so the error per partial stays far below
// 2^-18 * sum|x||w| (the bound the reference states for its three-term bf16 split).
//
// Used below 128 tokens, where the product is latency: 3.1 MB of gate, 12 KB of x per token. A CTA owns 16 experts x one K
// split x 16 tokens, so one token alone already spreads the gate over 128 CTAs (with 16 splits) of 24 KB each; every lane's
// gate values go to registers in one batch of independent 16-byte loads, issued before the wait for the predecessor's x.
// Bound by that one round trip up to about 16 tokens, by FMA issue above. Measured with both quantisers, us back to back:
// 2.5 / 3.7 / 4.5 / 8.6 / 13.7 at 1 / 16 / 32 / 64 / 100 tokens. The form before this one gave a CTA all 128 experts of one
// K split (16 CTAs, gate and x through 32-element shared-memory tiles, a barrier pair and a memory round trip per tile) and
// took 87 us at 1 token and 111 at 100.
#include "common.cuh"

namespace b200moe {

constexpr int kRgTokens = 16;             // tokens per CTA, 8 per warp
constexpr int kRgExperts = 16;            // experts per CTA, 4 per warp
constexpr int kRgChunk = 384;             // K elements in registers at a time: 3 x 4 per lane
constexpr int kRgRow = kRgChunk / 8;      // 16-byte vectors of a token's chunk in shared memory

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

// One step of the transposing sum over the lanes: before it, N values per lane; after it N / 2, the lanes with BIT clear
// holding the sums of the lower half and the others those of the upper half.
template <int N, int BIT>
__device__ __forceinline__ void fold_lanes(float* v, int lane) {
  const bool up = (lane & BIT) != 0;
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const float keep = up ? v[i + N / 2] : v[i], give = up ? v[i] : v[i + N / 2];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, BIT);
  }
}

// 16 bytes from an address that need not be aligned (`vec`: it is)
__device__ __forceinline__ float4 load_f32x4(const float* p, bool vec) {
  return vec ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(p[0], p[1], p[2], p[3]);
}
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

// grid (ceil(E / 16), S, ceil(T / 16)); warp w: experts 4 (w % 4) .. + 3, tokens 8 (w / 4) .. + 7 of the CTA's; the 32
// lanes share K, lane L holding elements 128 c + 4 L .. + 3 of every chunk.
template <bool QUANT>
__global__ void __launch_bounds__(256) router_gemm_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const float* __restrict__ gate, int64_t tokens,
                                                          int num_experts, int k_per_split,
                                                          float* __restrict__ partials, QuantOut q, bool vec) {
  __shared__ uint4 xs[kRgTokens][kRgRow];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int e0 = blockIdx.x * kRgExperts + 4 * (warp & 3), th = 8 * (warp >> 2);
  const int64_t t0 = static_cast<int64_t>(blockIdx.z) * kRgTokens;
  const int nt = static_cast<int>(min(static_cast<int64_t>(kRgTokens), tokens - t0));
  const int k0 = blockIdx.y * k_per_split;
  float4 g[3][4];
  auto load_gate = [&](int kk) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = kk + 128 * c + 4 * lane;
        g[c][j] = k < k_per_split && e0 + j < num_experts
                      ? load_f32x4(gate + static_cast<int64_t>(e0 + j) * kH + k0 + k, vec)
                      : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
  };
  load_gate(0);  // weights: no kernel of this library that lets its successor start early writes them
  pdl_enter(x);
  float acc[32];  // [token 0..7][expert 0..3]
#pragma unroll
  for (int i = 0; i < 32; ++i) acc[i] = 0.0f;
  for (int kk = 0; kk < k_per_split; kk += kRgChunk) {
    const int vecs = min(kRgChunk, k_per_split - kk) / 8;  // 16-byte vectors of a row in this chunk
    if (kk) {
      load_gate(kk);
      __syncthreads();
    }
    for (int i = tid; i < nt * kRgRow; i += 256) {
      const int r = i / kRgRow, c = i % kRgRow;
      xs[r][c] = c < vecs ? load_bf16x8(x + (t0 + r) * kH + k0 + kk + 8 * c, vec) : make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    if (QUANT) {
      // one pass over x: the CTAs of the expert groups share the chunk's blocks of 32 values; 4 threads x 8 values per block
      const int groups = gridDim.x, mine = (nt - static_cast<int>(blockIdx.x) + groups - 1) / groups;  // tokens of this CTA
      const int blocks = vecs / 4;
      for (int i = tid; i < ((mine * blocks * 4 + 31) & ~31); i += 256) {  // whole warps stay together for the shuffles
        const bool live = i < mine * blocks * 4;
        const int r = live ? (i / (blocks * 4)) * groups + static_cast<int>(blockIdx.x) : 0, v8 = live ? i % (blocks * 4) : 0;
        const uint4 raw = xs[r][v8];
        const uint32_t rr[4] = {raw.x, raw.y, raw.z, raw.w};
        float v[8];
        float amax = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[2 * j] = __uint_as_float(rr[j] << 16);
          v[2 * j + 1] = __uint_as_float(rr[j] & 0xffff0000u);
          amax = fmaxf(amax, fmaxf(fabsf(v[2 * j]), fabsf(v[2 * j + 1])));
        }
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
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      if (th + t < nt) {  // the same for the whole warp
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const uint2 b = reinterpret_cast<const uint2*>(&xs[th + t][0])[32 * c + lane];
          const float x0 = __uint_as_float(b.x << 16), x1 = __uint_as_float(b.x & 0xffff0000u);
          const float x2 = __uint_as_float(b.y << 16), x3 = __uint_as_float(b.y & 0xffff0000u);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float a = acc[4 * t + j];
            a = fmaf(x0, g[c][j].x, a);
            a = fmaf(x1, g[c][j].y, a);
            a = fmaf(x2, g[c][j].z, a);
            acc[4 * t + j] = fmaf(x3, g[c][j].w, a);
          }
        }
      }
    }
  }
  if (th >= nt) return;
  // 32 sums over the 32 lanes in 31 shuffles: lane L ends with entry L = token L / 4, expert L % 4
  fold_lanes<32, 16>(acc, lane);
  fold_lanes<16, 8>(acc, lane);
  fold_lanes<8, 4>(acc, lane);
  fold_lanes<4, 2>(acc, lane);
  fold_lanes<2, 1>(acc, lane);
  const int64_t t = t0 + th + (lane >> 2);
  const int e = e0 + (lane & 3);
  if (t < tokens && e < num_experts) partials[(static_cast<int64_t>(blockIdx.y) * tokens + t) * num_experts + e] = acc[0];
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
  B200MOE_LAUNCH(router_gemm_kernel<false>, grid, 256, 0, static_cast<cudaStream_t>(stream),
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
  B200MOE_LAUNCH(router_gemm_kernel<true>, grid, 256, 0, static_cast<cudaStream_t>(stream),
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
