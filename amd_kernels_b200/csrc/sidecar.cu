// The compact prepared input: the routed experts' FP4 codes are not sent; the receiver rebuilds them bit for bit from the
// shared expert's FP8 codes of the same row, both scale rows and one correction bit per value.
// candidate(v) = the FP4 code of |e4m3(v)| / 2^(s4 - s8) with the thresholds .25 .75 1.25 1.75 2.5 3.5 5 (ties to the even
// code), sign from the FP8 byte; mask bit = (candidate != direct code).
#include "common.cuh"

namespace b200moe {

// The candidate codes of 8 FP8 values, one nibble each: the FP8 values are exact in fp32, scaling by 2^(s8 - s4) is exact, and the
// hardware's round-to-nearest-even E2M1 conversion has exactly these thresholds.
// (Comparing against the seven thresholds value by value made the two kernels arithmetic-bound: 20 and 25 us at 2048 tokens.)
__device__ __forceinline__ void e4m3_pair(uint32_t codes, float& lo, float& hi) {
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(static_cast<uint16_t>(codes)));
  asm("{\n.reg .f16 a, b;\nmov.b32 {a, b}, %2;\ncvt.f32.f16 %0, a;\ncvt.f32.f16 %1, b;\n}\n" : "=f"(lo), "=f"(hi) : "r"(h2));
}
__device__ __forceinline__ uint32_t candidate_codes(const uint2 b8, float inv_ratio) {
  uint32_t out = 0;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float lo, hi;
    e4m3_pair((p < 2 ? b8.x : b8.y) >> (16 * (p & 1)), lo, hi);
    out |= cvt_e2m1x2(lo * inv_ratio, hi * inv_ratio) << (8 * p);
  }
  return out;
}
// the magnitude, in FP4 units, of the FP8 value in the low byte
__device__ __forceinline__ float magnitude(uint32_t code, float inv_ratio) {
  float lo, hi;
  e4m3_pair(code & 0xffu, lo, hi);
  return fabsf(lo * inv_ratio);
}

__device__ __forceinline__ float inverse_ratio(const uint8_t* s4, const uint8_t* s8, uint32_t block) {
  const int d = static_cast<int>(__ldcg(s8 + block)) - static_cast<int>(__ldcg(s4 + block));
  return __uint_as_float(static_cast<uint32_t>(min(max(d, -126), 127) + 127) << 23);  // 2^(s8 - s4), exact
}

// One thread = one 32-value block = one mask word: 32 FP8 codes, 16 bytes of FP4 codes, both scale bytes, read once per block. One
// thread per 8 values, with a byte of mask each, took 9.4 and 13.7 us at 2048 tokens; 32 values take 6.3 and 11.4, in which the scale
// atoms, once a launch of 3.4 us of their own, are included. A block's FP8 codes are read as two or four vectors, so that operands
// aligned to 8 bytes only are taken as before (`wide` false).
// Neither kernel launches its successor early: with 32 values to a thread their CTAs are all resident up to about 1500 tokens, the
// launches behind them followed at once, and at decode sizes GEMM1's first requests for weights ran beside the unpack and the gather,
// whose loads queue behind them (unpack 7.3 us at 400 tokens instead of 4.0). The prepared call, launch early / behind, us: 192.9 / 188.0
// at 257 tokens, 223.8 / 217.2 at 400, 253.1 / 246.6 at 480, 214.3 / 209.2 at 512, 231.9 / 226.6 at 777, 293.0 / 290.0 at 2048.
__device__ __forceinline__ void load_codes8(const uint8_t* q8, uint32_t block, bool wide, uint2 (&v)[4]) {
  if (wide) {
    const uint4* p = reinterpret_cast<const uint4*>(q8) + 2 * static_cast<int64_t>(block);
    const uint4 a = __ldcg(p), b = __ldcg(p + 1);
    v[0] = make_uint2(a.x, a.y);
    v[1] = make_uint2(a.z, a.w);
    v[2] = make_uint2(b.x, b.y);
    v[3] = make_uint2(b.z, b.w);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = __ldcg(reinterpret_cast<const uint2*>(q8) + 4 * static_cast<int64_t>(block) + k);
  }
}

__global__ void __launch_bounds__(256) sidecar_pack_kernel(const uint8_t* __restrict__ q4, const uint8_t* __restrict__ s4,
                                                           const uint8_t* __restrict__ q8, const uint8_t* __restrict__ s8,
                                                           uint32_t n_blocks, bool wide, uint32_t* __restrict__ mask) {
  pdl_wait();
  launder(q4), launder(s4), launder(q8), launder(s8);
  const uint32_t i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n_blocks) return;
  uint2 v8[4];
  load_codes8(q8, i, wide, v8);
  uint32_t v4[4];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint2 v = __ldcg(reinterpret_cast<const uint2*>(q4) + 2 * static_cast<int64_t>(i) + k);
    v4[2 * k] = v.x;
    v4[2 * k + 1] = v.y;
  }
  const float inv = inverse_ratio(s4, s8, i);
  uint32_t bits = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    uint32_t d = candidate_codes(v8[k], inv) ^ v4[k];
    d |= d >> 2;
    d = (d | d >> 1) & 0x11111111u;  // one bit per nibble that differs, then the eight bits side by side
    d = (d | d >> 3) & 0x03030303u;
    d = (d | d >> 6) & 0x000f000fu;
    bits |= ((d | d >> 12) & 0xffu) << (8 * k);
  }
  mask[i] = bits;
}

// `atoms` (may be null): the FP8 scales' atoms of blocks of 2^atom_shift rows as well, which the shared expert reads
__global__ void __launch_bounds__(256) sidecar_unpack_kernel(const uint32_t* __restrict__ mask, const uint8_t* __restrict__ s4,
                                                             const uint8_t* __restrict__ q8, const uint8_t* __restrict__ s8,
                                                             uint32_t n_blocks, bool wide, uint2* __restrict__ q4,
                                                             uint8_t* __restrict__ atoms, int atom_shift) {
  pdl_wait();
  launder(mask), launder(s4), launder(q8), launder(s8);
  const uint32_t i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n_blocks) return;
  if (atoms != nullptr && (i & 3u) == 0u) {
    const uint32_t row = i / (kH / 32);
    QuantRow8{nullptr, nullptr, atoms, atom_shift}.store_scales(row, static_cast<int>((i % (kH / 32)) >> 2),
                                                                __ldcg(reinterpret_cast<const uint32_t*>(s8) + (i >> 2)));
  }
  const uint32_t bits = __ldcg(mask + i);
  uint2 v8[4];
  load_codes8(q8, i, wide, v8);
  const float inv = inverse_ratio(s4, s8, i);
  uint32_t out[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    out[k] = candidate_codes(v8[k], inv);
    for (uint32_t m = (bits >> (8 * k)) & 0xffu; m != 0u; m &= m - 1u) {  // few values differ: one step per set bit
      // the other neighbour: below at the midpoints that round up (.75, 1.75, 3.5), above elsewhere
      const int j = __ffs(static_cast<int>(m)) - 1;
      const float v = magnitude((j < 4 ? v8[k].x : v8[k].y) >> (8 * (j & 3)), inv);
      const uint32_t step = v == 0.75f || v == 1.75f || v == 3.5f ? 7u : 1u;
      const uint32_t code = (out[k] >> (4 * j)) & 7u;
      out[k] ^= (code ^ ((code + step) & 7u)) << (4 * j);
    }
  }
  q4[2 * static_cast<int64_t>(i)] = make_uint2(out[0], out[1]);
  q4[2 * static_cast<int64_t>(i) + 1] = make_uint2(out[2], out[3]);
}

// row-major scale bytes [tokens][cols] -> the scale atoms of bm-row blocks [ceil(tokens/bm)][cols/4][512]; rows of the
// last block beyond `tokens` get the scale byte 1
__global__ void __launch_bounds__(256) scales_to_atoms_kernel(const uint8_t* __restrict__ rows, int64_t tokens, int cols,
                                                              int bm_shift, int64_t padded_rows, uint8_t* __restrict__ atoms) {
  pdl_enter(rows);
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;  // one 4-byte cell: (row, cols/4)
  const int cells = cols >> 2;
  if (i >= padded_rows * cells) return;
  const int64_t row = i / cells;
  const int a = static_cast<int>(i % cells);
  const uint32_t v = row < tokens ? __ldcg(reinterpret_cast<const uint32_t*>(rows + row * cols + 4 * a)) : 0x01010101u;
  const int r = static_cast<int>(row & ((1 << bm_shift) - 1));
  *reinterpret_cast<uint32_t*>(atoms + ((row >> bm_shift) * cells + a) * kAtomBytes + atom_offset(r, 0)) = v;
}

}  // namespace b200moe

static int sidecar_args(const void* a, const void* b, const void* c, const void* d, const void* e, int64_t tokens) {
  if (!a || !b || !c || !d || !e || tokens < 0 || tokens > B200MOE_MAX_TOKENS) return B200MOE_E_ARG;
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(e)) & 7)
    return B200MOE_E_ALIGN;
  return 0;
}

extern "C" int b200moe_sidecar_pack(const uint8_t* q4, const uint8_t* s4, const uint8_t* q8, const uint8_t* s8,
                                    int64_t tokens, uint8_t* mask, void* stream) {
  using namespace b200moe;
  const int r = sidecar_args(q4, s4, q8, s8, mask, tokens);
  if (r || tokens == 0) return r;
  const int64_t n = tokens * (kH / 32);
  B200MOE_LAUNCH(sidecar_pack_kernel, static_cast<unsigned>((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream), q4, s4, q8,
                 s8, static_cast<uint32_t>(n), (reinterpret_cast<uintptr_t>(q8) & 15) == 0, reinterpret_cast<uint32_t*>(mask));
  return 0;
}

namespace b200moe {
// b200moe_sidecar_unpack, and (atoms not null) the scale atoms of s8 in blocks of bm rows, rows beyond `tokens` left alone
int sidecar_unpack_atoms(const uint8_t* mask, const uint8_t* s4, const uint8_t* q8, const uint8_t* s8, int64_t tokens, uint8_t* q4,
                         uint8_t* atoms, int bm, void* stream) {
  const int r = sidecar_args(mask, s4, q8, s8, q4, tokens);
  if (r || tokens == 0) return r;
  if (atoms && ((reinterpret_cast<uintptr_t>(s8) & 3) || (reinterpret_cast<uintptr_t>(atoms) & 15))) return B200MOE_E_ALIGN;
  const int shift = bm == 16 ? 4 : bm == 32 ? 5 : bm == 64 ? 6 : 7;
  const int64_t n = tokens * (kH / 32);
  B200MOE_LAUNCH(sidecar_unpack_kernel, static_cast<unsigned>((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream),
                 reinterpret_cast<const uint32_t*>(mask), s4, q8, s8, static_cast<uint32_t>(n),
                 (reinterpret_cast<uintptr_t>(q8) & 15) == 0, reinterpret_cast<uint2*>(q4), atoms, shift);
  return 0;
}
}  // namespace b200moe

extern "C" int b200moe_sidecar_unpack(const uint8_t* mask, const uint8_t* s4, const uint8_t* q8, const uint8_t* s8,
                                      int64_t tokens, uint8_t* q4, void* stream) {
  return b200moe::sidecar_unpack_atoms(mask, s4, q8, s8, tokens, q4, nullptr, 16, stream);
}

extern "C" int b200moe_scales_to_atoms(const uint8_t* rows, int64_t tokens, int cols, int bm, uint8_t* atoms, void* stream) {
  using namespace b200moe;
  if (!rows || !atoms || tokens < 1 || tokens > B200MOE_MAX_TOKENS || cols < 4 || (cols & 3)) return B200MOE_E_ARG;
  const int shift = bm == 16 ? 4 : bm == 32 ? 5 : bm == 64 ? 6 : bm == 128 ? 7 : -1;
  if (shift < 0) return B200MOE_E_ARG;
  if ((reinterpret_cast<uintptr_t>(rows) & 3) || (reinterpret_cast<uintptr_t>(atoms) & 15)) return B200MOE_E_ALIGN;
  const int64_t padded = (tokens + bm - 1) / bm * bm;
  const int64_t n = padded * (cols >> 2);
  B200MOE_LAUNCH(scales_to_atoms_kernel, static_cast<unsigned>((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream), rows,
                 tokens, cols, shift, padded, atoms);
  return 0;
}
