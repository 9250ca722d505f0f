// GPU quantize + pack: bf16 W [N, K] -> int4 [N, K/2] + fp16 scales [N, K/128],
// bit-exact with CUDALM's offline quantizer (tools/common/w4a16_quant.py:25-60).
//
// Eight lanes own one group of 128 values, sixteen values each.  The arithmetic is the
// quantizer's: scale32 = amax / 7 (IEEE fp32), q = round-half-even(fl(w / scale32)) with
// the IEEE fp32 quotient, clamp to [-7, 7]; a group whose fp32 scale is zero stores q = 0;
// the stored scale is fp16_rn(scale32), which may be zero although q is not.
//
// Bound by DRAM traffic as long as a value costs few instructions (254 M values against
// 36 T lane-instructions per second are 7 us per instruction; the traffic of a
// 248320 x 1024 matrix is 99 us at the copy rate).  So:
//   * the quotients come from packed two-value arithmetic (fma.rn.f32x2) without a branch,
//     see quotients(); the group maximum from packed bf16 maxima of magnitudes;
//   * the eight codes of a word are put together in floating point, see pack_codes();
//   * a warp takes sixteen consecutive groups (4 KB of input) at a time with all its loads
//     in flight, writes whole 32-byte sectors of codes and 32 bytes of scales.
// Sixteen lanes per group, a branch to an exact divide near rounding boundaries and one
// bit-field insert per value took 10 instructions per value: 194 us for 248320 x 1024
// (3.29 TB/s of traffic); now 112 us call by call, 96 us replayed from a graph (5.7 and
// 6.7 TB/s).
#include "common.cuh"

namespace cb200 {

constexpr int kQuantThreads = 256;
constexpr int kGroupsPerTrip = 16;   // consecutive groups of a warp
constexpr int kLanesPerGroup = 8;
constexpr int kSubs = kGroupsPerTrip * kLanesPerGroup / 32;  // groups of a lane per trip

// ---- two fp32 values in one 64-bit register -----------------------------------------
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float* lo, float* hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(*lo), "=f"(*hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// the larger magnitude of each half (NaN if either is); the signs of the result are arbitrary
__device__ __forceinline__ std::uint32_t max_abs_bf16x2(std::uint32_t a, std::uint32_t b) {
  std::uint32_t r;
  asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// Range of scales for which the residuals of quotients() and of the scale's own division
// are exact (no underflow) and the reciprocal is a normal number.
constexpr float kScaleLo = 0x1p-90f, kScaleHi = 0x1p90f;

// rint(fl(w / s)) of two values, with inv = fl(1 / s): q0 = w * inv is within two ulps of
// the quotient, its residual is exact in one FMA, and a second FMA gives the correctly
// rounded quotient (Markstein's theorem on division with a fused multiply-add).  Where the
// integer rounding could be sensitive to the last bit -- 14 |w| an odd multiple of the
// group's maximum, at most 8 significant bits each -- the result was compared with the
// divide for every pair of significands and every exponent difference that matters.
__device__ __forceinline__ unsigned long long quotients(unsigned long long w, unsigned long long neg_s,
                                                        unsigned long long inv) {
  const unsigned long long q0 = mul2(w, inv);
  const unsigned long long rem = fma2(neg_s, q0, w);
  const unsigned long long q = fma2(rem, inv, q0);
  // adding and subtracting 1.5 * 2^23 rounds to the nearest integer, ties to even
  constexpr float kMagic = 12582912.0f;
  return add2(add2(q, pack2(kMagic, kMagic)), pack2(-kMagic, -kMagic));
}

// Eight integers q_0 .. q_7 in [-7, 7] (pairs {q_2i, q_2i+1}) as nibbles of a word, two's
// complement: sum of (q_i + 8) 16^i has no borrows between the fields, four of them are
// exact in fp32, and flipping bit 3 of each field turns q + 8 into two's complement.
__device__ __forceinline__ std::uint32_t pack_codes(const unsigned long long (&q)[4]) {
  const unsigned long long c256 = pack2(256.0f, 256.0f);
  float lo, hi;
  unpack2(fma2(q[1], c256, q[0]), &lo, &hi);
  const float a = fmaf(hi, 16.0f, lo) + (12582912.0f + 34952.0f);  // 34952 = 0x8888
  unpack2(fma2(q[3], c256, q[2]), &lo, &hi);
  const float b = fmaf(hi, 16.0f, lo) + (12582912.0f + 34952.0f);
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x5410) ^ 0x88888888u;
}

// A group whose scale lies outside [kScaleLo, kScaleHi] (a NaN among its values included,
// which the maximum ignores): IEEE divides, value by value.  The group's lanes call together.
__device__ __noinline__ uint2 quantize_slow(uint4 v0, uint4 v1, unsigned mask, float* scale_out) {
  const std::uint32_t words[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    amax = fmaxf(amax, fmaxf(fabsf(__uint_as_float(words[i] << 16)), fabsf(__uint_as_float(words[i] & 0xFFFF0000u))));
#pragma unroll
  for (int off = kLanesPerGroup / 2; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(mask, amax, off));
  const float s = __fdiv_rn(amax, 7.0f);
  *scale_out = s;
  std::uint32_t out[2] = {0u, 0u};
  if (s != 0.f) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float w = __uint_as_float((i & 1) ? (words[i >> 1] & 0xFFFF0000u) : (words[i >> 1] << 16));
      // No clamp: |w| <= amax and s = fl(amax / 7) >= (amax / 7)(1 - 2^-24) (for a
      // subnormal scale: within 2^-14 of it, the smallest bf16 being 2^-133), so the
      // quotient stays below 7.5 and rounds into [-7, 7] by itself.
      const float q = rintf(__fdiv_rn(w, s));
      out[i >> 3] |= (__float_as_uint(q + 12582912.0f) & 15u) << (4 * (i & 7));
    }
  }
  return make_uint2(out[0], out[1]);
}

// A lane's sixteen values of one group: two packed words and the group's scale.
__device__ __forceinline__ uint2 quantize_sixteen(const uint4 (&v)[2], unsigned mask, float* scale_out) {
  std::uint32_t m = max_abs_bf16x2(max_abs_bf16x2(max_abs_bf16x2(v[0].x, v[0].y), max_abs_bf16x2(v[0].z, v[0].w)),
                                   max_abs_bf16x2(max_abs_bf16x2(v[1].x, v[1].y), max_abs_bf16x2(v[1].z, v[1].w)));
#pragma unroll
  for (int off = kLanesPerGroup / 2; off > 0; off >>= 1) m = max_abs_bf16x2(m, __shfl_xor_sync(mask, m, off));
  // as integers, so that a NaN is the largest
  const float amax = __uint_as_float(max((m << 16) & 0x7FFF0000u, m & 0x7FFF0000u));
  const float s = __fdiv_rn(amax, 7.0f);
  *scale_out = s;
  if (!(s >= kScaleLo && s <= kScaleHi)) return quantize_slow(v[0], v[1], mask, scale_out);
  const float inv_s = __frcp_rn(s);
  const unsigned long long neg_s = pack2(-s, -s), inv = pack2(inv_s, inv_s);
  std::uint32_t out[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const std::uint32_t words[4] = {v[h].x, v[h].y, v[h].z, v[h].w};
    unsigned long long q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      q[i] = quotients(pack2(__uint_as_float(words[i] << 16), __uint_as_float(words[i] & 0xFFFF0000u)), neg_s, inv);
    out[h] = pack_codes(q);
  }
  return make_uint2(out[0], out[1]);
}

// 16-byte word (of a group's sixteen) of lane `l` of the group in load h: l + 8 h, so that a
// load covers 128 contiguous bytes of each of the warp's four groups, and the codes of one
// load are a whole 32-byte sector.
// One trip per warp and as many CTAs as that takes: the block scheduler's hand-out keeps
// DRAM busier than a resident grid that loops (248320 x 1024: 96.3 us against 104 us with
// four CTAs per SM, and 107 us at one register budget less).
__global__ void __launch_bounds__(kQuantThreads, 4)
quantize_w4a16_kernel(const uint4* __restrict__ W, std::uint32_t* __restrict__ packed,
                      std::uint16_t* __restrict__ scales, long long n_groups) {
  const int lane = threadIdx.x & 31;
  const int l = lane & (kLanesPerGroup - 1), octet = lane / kLanesPerGroup;
  const unsigned mask = 0xFFu << (octet * kLanesPerGroup);  // the lanes that share a group
  const long long g0 =
      ((static_cast<long long>(blockIdx.x) * kQuantThreads + threadIdx.x) >> 5) * kGroupsPerTrip;
  if (g0 + kGroupsPerTrip <= n_groups) {
    uint4 v[kSubs][2];
#pragma unroll
    for (int u = 0; u < kSubs; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) v[u][h] = __ldcs(W + (g0 + u * 4 + octet) * 16 + l + 8 * h);
    float mine = 0.f;  // the scale this lane stores: of group 4 l + octet of the trip
#pragma unroll
    for (int u = 0; u < kSubs; ++u) {
      const long long g = g0 + u * 4 + octet;
      float s;
      const uint2 out = quantize_sixteen(v[u], mask, &s);
      __stcs(packed + g * 16 + l, out.x);
      __stcs(packed + g * 16 + l + 8, out.y);
      if (l == u) mine = s;
    }
    if (l < kSubs) scales[g0 + l * 4 + octet] = __half_as_ushort(__float2half_rn(mine));
    return;
  }
  // the last warp's partial trip
  for (int u = 0; u < kSubs; ++u) {
    const long long g = g0 + u * 4 + octet;
    if (g >= n_groups) break;
    const uint4 v[2] = {__ldcs(W + g * 16 + l), __ldcs(W + g * 16 + l + 8)};
    float s;
    const uint2 out = quantize_sixteen(v, mask, &s);
    packed[g * 16 + l] = out.x;
    packed[g * 16 + l + 8] = out.y;
    if (l == 0) scales[g] = __half_as_ushort(__float2half_rn(s));
  }
}

}  // namespace cb200

extern "C" int cudalm_b200_quantize_w4a16(const uint16_t* w_bf16, int N, int K, uint8_t* packed,
                                          uint16_t* scales, void* stream) {
  using namespace cb200;
  if (!w_bf16 || !packed || !scales) return CUDALM_B200_ERR_NULL;
  if (N < 1 || K <= 0 || (K % 128) != 0) return CUDALM_B200_ERR_BAD_SHAPE;
  if (!aligned_to(w_bf16, 16) || !aligned_to(packed, 4)) return CUDALM_B200_ERR_MISALIGNED;
  const long long n_groups = static_cast<long long>(N) * (K / 128);
  const long long warps = (n_groups + kGroupsPerTrip - 1) / kGroupsPerTrip;
  const long long blocks = (warps + kQuantThreads / 32 - 1) / (kQuantThreads / 32);
  if (blocks > 0x7fffffffll) return CUDALM_B200_ERR_TOO_LARGE;
  quantize_w4a16_kernel<<<static_cast<int>(blocks), kQuantThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const uint4*>(w_bf16), reinterpret_cast<std::uint32_t*>(packed), scales,
      n_groups);
  return check_launch();
}
