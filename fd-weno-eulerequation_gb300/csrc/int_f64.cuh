// FP64 products, reciprocals and quotients on the integer pipes, each rounded
// to nearest even exactly as the FP64 instruction would.
//
// Why: the parity path is bound by the FP64 pipe, which takes about 19 cycles
// of an SM per warp instruction (1.06 TFLOP/s over 152 SMs), the room of about
// 76 instructions of the four schedulers, while they issue on 7 % of their
// cycles.  A product here is about 30 integer instructions, a reciprocal about
// 50 and a further quotient by the same divisor about 30 (an IEEE division is
// about 7.5 FP64 operations), so products and quotients leave the FP64 pipe to
// the sums and run beside them.
//
// Domain: operands are zeros or normal numbers and no result overflows or is
// subnormal (int_mul_ftz: a subnormal result becomes zero).  Callers test the
// ranges (in_range) and take FP64 arithmetic elsewhere.  The sign of a zero
// result is not kept (a zero comes out as +0).
#pragma once

namespace wenofd {
namespace dev {

#ifdef __CUDACC__
#define WENOFD_HD __host__ __device__ __forceinline__
#else
#define WENOFD_HD inline
#endif

typedef unsigned int u32;
typedef unsigned long long u64;

WENOFD_HD u64 f64_bits(double x) {
#ifdef __CUDA_ARCH__
  return u64(__double_as_longlong(x));
#else
  u64 u;
  __builtin_memcpy(&u, &x, 8);
  return u;
#endif
}
WENOFD_HD double bits_f64(u32 hi, u32 lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(int(hi), int(lo));
#else
  const u64 u = (u64(hi) << 32) | lo;
  double x;
  __builtin_memcpy(&x, &u, 8);
  return x;
#endif
}
// the low word of (hi:lo) >> s, s in [1, 31]
WENOFD_HD u32 shr_lo(u32 hi, u32 lo, u32 s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, s);
#else
  return (lo >> s) | (hi << (32 - s));
#endif
}
WENOFD_HD u64 mul_hi64(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return u64((static_cast<unsigned __int128>(a) * b) >> 64);
#endif
}
WENOFD_HD float rcp_seed(float x) {  // relative error below 2^-22
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / x;
#endif
}
WENOFD_HD float rsqrt_seed(float x) {  // relative error below 2^-22
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / __builtin_sqrtf(x);
#endif
}
WENOFD_HD u32 float_bits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  u32 u;
  __builtin_memcpy(&u, &x, 4);
  return u;
#endif
}
WENOFD_HD float bits_float(u32 u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  __builtin_memcpy(&x, &u, 4);
  return x;
#endif
}

// A seed in [1/2, 1) as 2^32 times itself.  The exact value lies in that interval,
// but an approximation may fall short of 1/2 by its error; unclamped, its exponent
// would be read as part of the fraction, off by a factor of two.  (At the upper
// end the callers keep clear of 1.)  2^8 times the bits drops the exponent field.
WENOFD_HD u32 seed_fixed(u32 bits) { return (bits < 0x3f000000u ? 0x3f000000u : bits) * 256u + 0x80000000u; }

// x is a zero or |x| in [2^lo, 2^hi) (exponents unbiased)
template <int LO, int HI>
WENOFD_HD bool in_range(double x) {
  const u64 u = f64_bits(x);
  const u32 mag = u32(u >> 32) & 0x7fffffffu;
  return mag - (u32(1023 + LO) << 20) < (u32(HI - LO) << 20) || (mag | u32(u)) == 0u;
}

// x is in [2^lo, 2^hi)
template <int LO, int HI>
WENOFD_HD bool positive_in_range(double x) {
  return u32(f64_bits(x) >> 32) - (u32(1023 + LO) << 20) < (u32(HI - LO) << 20);
}

// x / 2, x a zero or at least 2^-1021 in magnitude
WENOFD_HD double int_half(double x) {
  const u64 u = f64_bits(x);
  const u32 hi = u32(u >> 32);
  return bits_f64((hi & 0x7ff00000u) == 0u ? hi : hi - 0x100000u, u32(u));
}

// a * b.  The product of the two 53-bit significands has 106 bits or 105; its
// top 53 are the result's and what lies below decides the rounding.  The
// exponent fields add with the sign bits above them, and the significand's
// leading 1 and a carry of the rounding add into the exponent field.
template <bool FTZ = false>
WENOFD_HD double int_mul(double a, double b) {
  const u64 ua = f64_bits(a), ub = f64_bits(b);
  const u32 ah = u32(ua >> 32), al = u32(ua), bh = u32(ub >> 32), bl = u32(ub);
  const u32 Ah = (ah & 0xfffffu) | 0x100000u, Bh = (bh & 0xfffffu) | 0x100000u;
  const u64 ll = u64(al) * bl;
  const u64 m = u64(al) * Bh + (u64(Ah) * bl + (ll >> 32));
  const u64 hh = u64(Ah) * Bh + (m >> 32);  // bits 64..105
  const u32 top = u32(hh >> 32), low = u32(hh), rest = u32(m);
  const u32 n = top >> 9;  // 1: 106 bits
  const u32 Rh = shr_lo(top, low, 20u + n), Rl = shr_lo(low, rest, 20u + n);
  const u32 c = (rest << (12u - n)) | (u32(ll) != 0u ? 1u : 0u);  // the bits below, the last one sticky
  const u32 ex = (ah & 0xfff00000u) + (bh & 0xfff00000u) - 0x40000000u + (n << 20);
  // up when c > 1/2, or c = 1/2 and the significand is odd
  const u32 up = u32((u64(c) + (0x7fffffffu + (Rl & 1u))) >> 32);
  const u64 R = ((u64(Rh + ex) << 32) | Rl) + up;
  bool zero = (ah & 0x7ff00000u) == 0u || (bh & 0x7ff00000u) == 0u;
  if (FTZ) {
    const int e = int((ah & 0x7ff00000u) + (bh & 0x7ff00000u)) - 0x40000000 + int(n << 20);
    zero = zero || e < 0;
  }
  return zero ? 0.0 : bits_f64(u32(R >> 32), u32(R));
}
WENOFD_HD double int_mul_ftz(double a, double b) { return int_mul<true>(a, b); }

// A positive normal divisor x = X 2^(e - 52), X its 53-bit significand, and
// Y = 2^116 / X to within a few units (62 bits or more): a 23-bit seed and two
// Newton steps in fixed point.
struct IntDivisor {
  u64 X, Y;
  u32 hi;  // x's exponent field
  WENOFD_HD explicit IntDivisor(double x) {
    const u64 u = f64_bits(x);
    hi = u32(u >> 32) & 0x7ff00000u;
    X = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    const u64 XL = X << 11;  // in [2^63, 2^64)
    const u32 xh = u32(XL >> 32), xl = u32(XL);
    // seed: 1 / (the leading 24 bits of the significand, rounded up by two), below
    // 1 whatever its error
    const float r = rcp_seed(bits_float(0x3f800002u + ((xh >> 8) & 0x7fffffu)));
    const u32 y0 = seed_fixed(float_bits(r));  // 2^32 / significand
    const u64 P = u64(xh) * y0 + ((u64(xl) * y0) >> 32);                   // 2^63 (1 - e)
    const int E = int((long long)(0x8000000000000000ull - P) >> 11);       // e 2^52
    const u64 Y1 = (u64(y0) << 32) + u64(((long long)(int(y0 >> 1)) * E) >> 19);
    const int D = int((long long)(0x8000000000000000ull - mul_hi64(XL, Y1)));  // the error left, 2^63
    Y = Y1 + u64(((long long)(int(u32(Y1 >> 33))) * D) >> 30);
  }
  // 1 / x: q = floor(2^105 / X) or one less, and one more where the exact
  // remainder says that 1/x lies above the midpoint q + 1/2 (a reciprocal or a
  // quotient never lies on one).  A power of two comes out as the carry.
  WENOFD_HD double reciprocal() const {
    const u64 q = (Y - 32) >> 11;
    const long long T = -(long long)(X * (2 * q + 1));  // 2^106 - X (2 q + 1)
    const u64 r = q + (T > 0 ? 1u : 0u);
    // q has its leading 1 in the exponent field: 2^-e-1 is 1023 - e - 1 there
    return bits_f64(u32(r >> 32) + (0x7fc00000u - hi), u32(r));
  }
  // a / x, a zero or normal
  WENOFD_HD double quotient(double a) const {
    const u64 u = f64_bits(a);
    const u32 ah = u32(u >> 32);
    const u64 A = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    const u64 Q = mul_hi64(A << 11, Y) - 32;  // 2^63 A / X, a little low
    const u32 s = u32(Q >> 63) ^ 1u;          // 1: A / X below 1
    const u64 q = (Q << s) >> 11;
    // A 2^(53 + s) - X (2 q + 1): its low 64 bits, and so its sign
    const long long T = (long long)((u64(u32(u) << (21u + s)) << 32) - X * (2 * q + 1));
    const u64 r = q + (T > 0 ? 1u : 0u);
    const u32 ex = (ah & 0xfff00000u) - hi + 0x3fe00000u - (s << 20);
    return (ah & 0x7ff00000u) == 0u ? 0.0 : bits_f64(u32(r >> 32) + ex, u32(r));
  }
};

// sqrt(x), x positive and normal.  With f = x's significand in [1, 4), even
// exponent: a 22-bit seed y of 1/sqrt(f) and two steps s += (f - s^2) y / 2 in
// fixed point, the first square exact, the second to 62 bits; then as in
// IntDivisor the root's 53 bits or one less, and the sign of the exact f - (q +
// 1/2)^2 (never zero).
WENOFD_HD double int_sqrt(double x) {
  const u64 u = f64_bits(x);
  const u32 hi = u32(u >> 32);
  const u32 odd = (~hi >> 20) & 1u;  // an even exponent field is an odd exponent
  const u64 M = ((u & 0xfffffffffffffull) | 0x10000000000000ull) << odd;  // f 2^52
  const u64 A = M << 10;                                                 // f 2^62
  const u32 f32 = (u32(u >> 29) & 0x7fffffu) + (odd ? 0x40000001u : 0x3f800001u);
  const u32 yb = float_bits(rsqrt_seed(bits_float(f32)));
  const u32 y = seed_fixed(yb < 0x3f7fffffu ? yb : 0x3f7fffffu);  // 2^32 / sqrt(f)
  const u32 s0 = u32((u64(u32(A >> 32)) * y) >> 32);                         // s 2^30
  const long long R0 = (long long)(A - ((u64(s0) * s0) << 2));               // (f - s^2) 2^62
  const u64 S1 = (u64(s0) << 32) + u64(((long long)int(R0 >> 13) * int(y >> 1)) >> 19);  // s 2^62
  const int R1 = int((long long)((A >> 2) - mul_hi64(S1, S1)));                          // (f - s^2) 2^60
  const u64 S = S1 + u64(((long long)R1 * int(y >> 1)) >> 30);
  const u64 q = (S - 32) >> 10;
  const u64 h = 2 * q + 1;
  const long long T = (long long)((u64(u32(M) << 22) << 32) - h * h);  // M 2^54 - h^2
  const u64 r = q + (T > 0 ? 1u : 0u);
  const u32 ex = ((hi & 0x7ff00000u) + 0x3ff00000u) >> 1;
  return bits_f64(u32(r >> 32) + (ex & 0x7ff00000u) - 0x100000u, u32(r));
}

}  // namespace dev
}  // namespace wenofd
