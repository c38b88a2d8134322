// szp_unpack.cuh -- unpacking and dequantizing pieces shared by the decoders.
#pragma once
#include "szp_device.cuh"
#include "szp_f64.h"

namespace szp {

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// (float)q * eb (szpd_float.cc:67,86,112).  NaN can only appear when eb is
// not finite; `special` (warp-uniform) selects the x86 NaN rule then.
__device__ __forceinline__ float dequant(uint32_t q, float eb, bool special = false) {
  float f = __int2float_rn((int32_t)q);
  float r = __fmul_rn(f, eb);
  return special ? x86_nan_fix(r, f, eb) : r;
}

// (double)q * eb for float64 streams (szpd_double.cc:67,86,112).
__device__ __forceinline__ double dequant(uint32_t q, double eb, bool special = false) {
  const double f = (double)(int32_t)q;
  const double r = __dmul_rn(f, eb);
  return special ? x86_nan_fix_d(r, f, eb) : r;
}

// (double)q * eb of float64 data as bits: integer arithmetic for every eb
// whose products stay normal (szp_f64.h), the FP64 multiply otherwise.
struct DequantD {
  uint64_t m, sgn;
  uint32_t ef;
  bool fast, special;
  double eb;
  __device__ __forceinline__ explicit DequantD(double e) : eb(e) {
    const uint64_t u = f64i::bits_of(e);
    fast = f64i::dequant_fast_ok(u);
    special = !isfinite(e);
    m = (u & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    ef = (uint32_t)(u >> 52) & 0x7FFu;
    sgn = u & 0x8000000000000000ull;
  }
  __device__ __forceinline__ unsigned long long operator()(uint32_t q) const {
    return fast ? f64i::dequant_bits((int32_t)q, m, ef, sgn) : f64i::bits_of(dequant(q, eb, special));
  }
};

// All ones when byte k of w has its top bit set, else 0 (prmt's sign
// replication; the __byte_perm intrinsic takes only the selector's low 3 bits).
__device__ __forceinline__ uint32_t prmt_sign(uint32_t w, int k) {
  uint32_t r;
  switch (k) {
    case 0: asm("prmt.b32 %0, %1, 0, 0x8888;" : "=r"(r) : "r"(w)); break;
    case 1: asm("prmt.b32 %0, %1, 0, 0x9999;" : "=r"(r) : "r"(w)); break;
    case 2: asm("prmt.b32 %0, %1, 0, 0xAAAA;" : "=r"(r) : "r"(w)); break;
    default: asm("prmt.b32 %0, %1, 0, 0xBBBB;" : "=r"(r) : "r"(w)); break;
  }
  return r;
}

// Little-endian bytes [o, o+8) of shared array b as (lo, hi), from three
// aligned 32-bit loads and two funnel shifts (reads b[o&~3 .. (o&~3)+12)).
__device__ __forceinline__ void lds_le64(const uint8_t* b, uint32_t o, uint32_t& lo, uint32_t& hi) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(b + (o & ~3u));
  const uint32_t sh = (o & 3u) * 8u;
  const uint32_t w0 = w[0], w1 = w[1], w2 = w[2];
  lo = __funnelshift_r(w0, w1, sh);
  hi = __funnelshift_r(w1, w2, sh);
}

// Little-endian bytes [o, o+4) (reads b[o&~3 .. (o&~3)+8)).
__device__ __forceinline__ uint32_t lds_le32(const uint8_t* b, uint32_t o) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(b + (o & ~3u));
  return __funnelshift_r(w[0], w[1], (o & 3u) * 8u);
}

// Little-endian bytes [o, o+16) (reads b[o&~3 .. (o&~3)+20)).
__device__ __forceinline__ void lds_le128(const uint8_t* b, uint32_t o, uint32_t (&w)[4]) {
  const uint32_t* p = reinterpret_cast<const uint32_t*>(b + (o & ~3u));
  const uint32_t sh = (o & 3u) * 8u;
  const uint32_t v[5] = {p[0], p[1], p[2], p[3], p[4]};
#pragma unroll
  for (int i = 0; i < 4; i++) w[i] = __funnelshift_r(v[i], v[i + 1], sh);
}

// sum + the products of a's unsigned and w's signed bytes.
__device__ __forceinline__ uint32_t dp4a_us(uint32_t a, uint32_t w, uint32_t sum) {
  uint32_t r;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(w), "r"(sum));
  return r;
}
// sum + the products of a's two unsigned 16-bit halves and w's signed bytes 0, 1 (HI: 2, 3).
template <bool HI>
__device__ __forceinline__ uint32_t dp2a_us(uint32_t a, uint32_t w, uint32_t sum) {
  uint32_t r;
  if (HI) {
    asm("dp2a.hi.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(w), "r"(sum));
  } else {
    asm("dp2a.lo.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(w), "r"(sum));
  }
  return r;
}

// The 8 deltas of lane `sub` of a full block of 8*LPB values (fastmode2: one
// fewer) whose bit-count byte is at s[o]; s is a 16-byte-aligned shared array.
// PL: the byte planes of the warp's blocks at most: 0, 1, 2, or 3 for any
// number.  A block of bit count 0 gives zeros (its lane reads bytes past it,
// which the caller has staged).
//
// The deltas are not taken apart.  Four remainder fields are spread to the
// bytes of a word (two multiply-adds move the upper fields up), their signs to
// bytes of +-1, and running sums are dot products with the weights masked to
// the first few bytes: about 5 instructions a value against 9 for shift, sign
// and add one by one, and half of them on the multiply pipe instead of the
// logic pipe that bounds these kernels.
template <int LPB, bool FM2, int PL>
struct Deltas {
  uint32_t x[2], w[2];       // value 4h + 3 - k in byte k: remainder field, weight
  uint32_t pl[PL == 1 ? 2 : PL == 2 ? 4 : 1];  // plane bytes in the same order; two planes: 16 bits per value, value order
  uint32_t pw;               // 1 << remainder bits
  uint32_t d[PL == 3 ? 8 : 1];
  uint32_t first4, total;    // sums of the first four deltas and of all

  __device__ __forceinline__ Deltas(const uint8_t* s, uint32_t o, uint32_t bc, int sub) {
    constexpr uint32_t MF = FM2 ? 8 * LPB - 1 : 8 * LPB;  // packed values; their sign bytes are LPB either way
    const uint32_t B = PL == 0 ? 0u : bc >> 3, rr = PL == 0 ? bc : bc & 7;
    const uint32_t sb = s[o + 1 + sub];  // sign bits, value 0 in bit 7 (szp_TypeManager.cc:820-844)
    uint32_t lo, hi;
    lds_le64(s, o + 1 + LPB + B * MF + rr * sub, lo, hi);
    const uint32_t t = __byte_perm(lo, 0, 0x0123);  // remainder bits, MSB first (szp_TypeManager.cc:122-434)
    const uint32_t t2 = __funnelshift_l(__byte_perm(hi, 0, 0x0123), t, 4 * rr);  // from value 4 on
    const uint32_t q8 = o + 1 + LPB + 8 * B * sub;  // the lane's plane bytes (szp_TypeManager.cc:36-52)
    pw = 1u << rr;
    if constexpr (PL == 3) {
      // byte k of sw has the sign bit of value k (4 + k) as its top bit
      const uint32_t sw[2] = {sb * 0x08040201u, (sb << 4) * 0x08040201u};
      const uint32_t mask = B >= 4 ? 0xFFFFFFFFu : (1u << (8 * B)) - 1u;
      total = 0;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const uint32_t h = lds_le32(s, q8 + j * B) & mask;
        // the plane bytes above the remainder bits, in one funnel shift
        const uint32_t v = __funnelshift_l((j < 4 ? t : t2) << (rr * (j & 3)), h, rr);
        const uint32_t sg = prmt_sign(sw[j >> 2], j & 3);  // 0 or all ones
        d[j] = (v ^ sg) - sg;
        total += d[j];
      }
    } else {
      const uint32_t k1 = 256u - pw, k2 = 65536u - pw * pw, m1 = pw * 0x00010001u - 0x00010001u;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        uint32_t v = __funnelshift_l(h ? t2 : t, 0u, 4 * rr);  // four fields, value 4h on top
        v = (v >> (2 * rr)) * k2 + v;          // two fields in each half
        x[h] = ((v >> rr) & m1) * k1 + v;      // one in each byte
        w[h] = (((h ? sb & 15u : sb >> 4) * 0x00204081u) & 0x01010101u) * 0xFEu + 0x01010101u;
      }
      first4 = dp4a_us(x[0], w[0], 0u);
      total = dp4a_us(x[1], w[1], first4);
      if constexpr (PL == 1) {
        uint32_t a, b;
        lds_le64(s, q8, a, b);
        pl[0] = B ? __byte_perm(a, 0, 0x0123) : 0u;
        pl[1] = B ? __byte_perm(b, 0, 0x0123) : 0u;
        const uint32_t h0 = dp4a_us(pl[0], w[0], 0u);
        first4 += h0 * pw;
        total += dp4a_us(pl[1], w[1], h0) * pw;
      }
      if constexpr (PL == 2) {
        uint32_t v[4];
        lds_le128(s, q8, v);
        const uint32_t se = B == 2 ? 0x3210u : B == 1 ? 0x4140u : 0x4444u, so = B == 1 ? 0x4342u : se;
        pl[0] = __byte_perm(v[0], 0, se);
        pl[1] = __byte_perm(B == 2 ? v[1] : v[0], 0, so);
        pl[2] = __byte_perm(B == 2 ? v[2] : v[1], 0, se);
        pl[3] = __byte_perm(B == 2 ? v[3] : v[1], 0, so);
        const uint32_t r0 = __byte_perm(w[0], 0, 0x0123), r1 = __byte_perm(w[1], 0, 0x0123);
        const uint32_t h0 = dp2a_us<true>(pl[1], r0, dp2a_us<false>(pl[0], r0, 0u));
        first4 += h0 * pw;
        total += dp2a_us<true>(pl[3], r1, dp2a_us<false>(pl[2], r1, h0)) * pw;
      }
    }
  }

  // q[j] = q0 + the first j deltas, j = 0..7.
  __device__ __forceinline__ void before(uint32_t q0, uint32_t (&q)[8]) const {
    q[0] = q0;
    if constexpr (PL == 3) {
#pragma unroll
      for (int j = 1; j < 8; j++) q[j] = q[j - 1] + d[j - 1];
      return;
    }
    q[4] = q0 + first4;
#pragma unroll
    for (int h = 0; h < 2; h++) {
#pragma unroll
      for (int j = 1; j < 4; j++) {
        const uint32_t wm = w[h] & (0xFFFFFFFFu << (32 - 8 * j));  // the first j values
        q[4 * h + j] = dp4a_us(x[h], wm, q[4 * h]);
        if constexpr (PL == 1) q[4 * h + j] += dp4a_us(pl[h], wm, 0u) * pw;
      }
      if constexpr (PL == 2) {
        const uint32_t r = __byte_perm(w[h], 0, 0x0123);
        const uint32_t h1 = dp2a_us<false>(pl[2 * h], r & 0xFFu, 0u), h2 = dp2a_us<false>(pl[2 * h], r, 0u);
        q[4 * h + 1] += h1 * pw;
        q[4 * h + 2] += h2 * pw;
        q[4 * h + 3] += dp2a_us<true>(pl[2 * h + 1], r & 0x00FFFFFFu, h2) * pw;
      }
    }
  }
};

// The 8 deltas of lane `sub` of a block of any m values: ml of them are the lane's (the others
// come out 0).
template <int LPB>
__device__ __forceinline__ void unpack_any(const uint8_t* s, uint32_t o, uint32_t bc, uint32_t m, uint32_t ml, int sub,
                                           uint32_t (&d)[8]) {
#pragma unroll
  for (int j = 0; j < 8; j++) d[j] = 0;
  if (bc == 0 || ml == 0) return;
  const uint32_t ns = (m + 7) >> 3, B = bc >> 3, rr = bc & 7;
  const uint32_t sb = s[o + 1 + sub];
  uint64_t acc = 0;  // 56-bit window: field j occupies bits [56 - rr*(j+1), 56 - rr*j)
  if (rr) {
    const uint8_t* rp = s + o + 1 + ns + B * m + rr * sub;
    const uint32_t nb = (ml * rr + 7) >> 3;
#pragma unroll
    for (uint32_t k = 0; k < 7; k++) acc = (acc << 8) | (uint64_t)(k < nb ? rp[k] : 0u);
  }
  const uint32_t mask = (1u << rr) - 1u;
  const uint8_t* q8 = s + o + 1 + ns + 8 * B * sub;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    if ((uint32_t)j < ml) {
      uint32_t h = 0;
      for (uint32_t b = 0; b < B; b++) h |= (uint32_t)q8[j * B + b] << (8 * b);
      const uint32_t v = (B ? h << rr : 0u) | (rr ? (uint32_t)(acc >> (56 - rr * (j + 1))) & mask : 0u);
      d[j] = ((sb >> (7 - j)) & 1u) ? 0u - v : v;
    }
  }
}

}  // namespace szp
