// Sums of doubles in integer arithmetic.
//
// On GB300 an FP64 add issues once per ~64 cycles and scheduler and takes
// ~150-180 cycles, so the ten dependent adds of a block or grid sum cost
// more than the memory round trips around them, while integer adds, shifts
// and the warp reductions (redux.sync) run at full rate.  A sum is taken in
// two passes: the largest exponent, then the values as 69-bit fixed-point
// numbers relative to it, in limbs whose 32-bit sums cannot overflow.
// Integer sums do not depend on the order; the only rounding is the cut at
// 2^-68 of the largest value per addend (an FP64 sum rounds every partial
// sum at 2^-53) and one rounding to nearest of the total.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gsls {

constexpr int kFixMask = (1 << 23) - 1;

__host__ __device__ __forceinline__ int fix_exp(unsigned long long bits) {
  return (int)((bits >> 52) & 0x7ffu);
}

// value = (S2 2^46 + S1 2^23 + S0) 2^(emax - 1091), |S_k| < 2^23 here; sums of
// up to 256 of them stay below 2^31
__host__ __device__ __forceinline__ void fix_limbs(unsigned long long bits, int emax, int S[3]) {
  const int e = fix_exp(bits);
  unsigned long long m = bits & 0xfffffffffffffull;
  m = e ? m | (1ull << 52) : m;
  const int sh = emax - (e ? e : 1);
  int s2 = 0, s1 = 0, s0 = 0;
  if (sh < 23) s2 = (int)(m >> (30 + sh));
  if (sh < 46) s1 = (int)((m >> (7 + sh)) & kFixMask);
  if (sh < 69) s0 = (int)((sh >= 16 ? m >> (sh - 16) : m << (16 - sh)) & kFixMask);
  const int sg = (int)((long long)bits >> 63);
  S[0] = (s0 ^ sg) - sg;
  S[1] = (s1 ^ sg) - sg;
  S[2] = (s2 ^ sg) - sg;
}

// hi 2^23 + lo, 0 <= lo < 2^23, shifted down by sh >= 0 bits with floor
__host__ __device__ __forceinline__ void fix_down(long long &hi, int &lo, int sh) {
  if (sh < 23) {
    lo = (int)((((unsigned long long)hi << (23 - sh)) & kFixMask) | (unsigned)(lo >> sh));
  } else {
    lo = (int)((hi >> (sh - 23 < 63 ? sh - 23 : 63)) & kFixMask);
  }
  hi >>= sh < 63 ? sh : 63;
}

// a block sum (e; S2, S1, S0) relative to E >= e: hi 2^23 + lo, 0 <= lo < 2^23,
// |hi| < 2^55 (shifted down with floor)
__host__ __device__ __forceinline__ void fix_align(int e, const int S[3], int E, long long &hi,
                                                   int &lo) {
  hi = (long long)S[2] * (1 << 23) + S[1] + (S[0] >> 23);
  lo = S[0] & kFixMask;
  fix_down(hi, lo, E - e);
}

// (hi 2^23 + lo) 2^(E - 1091) rounded to nearest; |hi| < 2^62, 0 <= lo < 2^31
__host__ __device__ __forceinline__ double fix_double(long long hi, unsigned lo, int E) {
  // carry, then sign and magnitude as H 2^23 + l
  hi += lo >> 23;
  int l = (int)(lo & kFixMask);
  const bool neg = hi < 0;
  unsigned long long H = (unsigned long long)hi;
  if (neg) {
    H = ~H;  // -(hi 2^23 + l) = (-hi - 1) 2^23 + (2^23 - l)
    l = (1 << 23) - l;
    if (l == (1 << 23)) {
      l = 0;
      H += 1;
    }
  }
  if (H == 0 && l == 0) return 0.0;
#ifdef __CUDA_ARCH__
  const int n = H ? 63 - __clzll((long long)H) : -1;
#else
  const int n = H ? 63 - __builtin_clzll(H) : -1;
#endif
  // the top bit of the number is bit n + 23; m: its leading 54 bits and a
  // sticky bit
  unsigned long long m;
  int top = n + 23;  // weight of the leading bit, in units of 2^(E - 1091)
  if (n >= 31) {     // at least 55 bits: drop n - 31 of H 2^23 + l
    const int d = n - 31;
    if (d >= 23) {
      m = H >> (d - 23);
      if ((H & ((1ull << (d - 23)) - 1)) || l) m |= 1;
    } else {
      m = (H << (23 - d)) | (unsigned long long)(l >> d);
      if (l & ((1 << d) - 1)) m |= 1;
    }
  } else {  // fewer: exact
    m = (H << 23) | (unsigned long long)l;
#ifdef __CUDA_ARCH__
    top = 63 - __clzll((long long)m);
#else
    top = 63 - __builtin_clzll(m);
#endif
    m <<= 54 - top;
  }
  // m has its leading bit at 54: 53 bits, a round bit and a sticky bit
  int ex = E - 1091 + top + 1023;  // biased exponent of the leading bit
  unsigned long long r;
  if (ex > 0) {
    r = (m >> 2) + (((m & 2) && (m & 5)) ? 1 : 0);
    if (r >> 53) {
      r >>= 1;
      ex++;
    }
    if (ex >= 0x7ff) r = 0x7ffull << 52;
    else r = ((unsigned long long)ex << 52) | (r & 0xfffffffffffffull);
  } else {  // subnormal: cut
    r = ex > -53 ? (m >> 2) >> (1 - ex) : 0ull;
  }
  r |= neg ? 1ull << 63 : 0ull;
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)r);
#else
  double d;
  __builtin_memcpy(&d, &r, 8);
  return d;
#endif
}

// high 64 bits of a 64 x 64-bit product
__host__ __device__ __forceinline__ unsigned long long fix_mulhi(unsigned long long a,
                                                                 unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
#endif
}

// a / b for the Krylov scalars, within 0.51 ulp, in integer arithmetic: the
// mantissa of 1/b by Newton's y <- y (2 - b y) in 64-bit fixed point from an
// FP32 start (2^-22, then 2^-44, then the last bits), times the mantissa of
// a.  The FP64 division takes ~2,500 cycles on one lane, this ~400.  Zeros,
// subnormals, infinities, NaN and results outside the normal range take the
// plain division.
__host__ __device__ __forceinline__ double fix_div(double a, double b) {
#ifdef __CUDA_ARCH__
  const unsigned long long ua = (unsigned long long)__double_as_longlong(a);
  const unsigned long long ub = (unsigned long long)__double_as_longlong(b);
#else
  unsigned long long ua, ub;
  __builtin_memcpy(&ua, &a, 8);
  __builtin_memcpy(&ub, &b, 8);
#endif
  const int ea = fix_exp(ua), eb = fix_exp(ub);
  int ex = ea - eb + 1023;
  if (ea == 0 || eb == 0 || ea == 0x7ff || eb == 0x7ff || ex < 2 || ex > 0x7fd) return a / b;
  // mantissas with the leading bit at 63: m / 2^64 in [1/2, 1)
  const unsigned long long A = ((ua & 0xfffffffffffffull) | (1ull << 52)) << 11;
  const unsigned long long B = ((ub & 0xfffffffffffffull) | (1ull << 52)) << 11;
  // y = 2^64 / B in (1, 2] as Y = y 2^62
  const float bf = (float)(unsigned)(B >> 40);  // 24 bits, exact
  float rf = 1.0f / bf;                         // y / 2^24
  unsigned long long Y = (unsigned long long)(rf * 9007199254740992.0f) << 33;  // 2^53
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const unsigned long long t = fix_mulhi(B, Y);      // b y 2^62, near 2^62
    Y = fix_mulhi(Y, (1ull << 63) - t) << 2;
  }
  // q = a y in (1/2, 2): Q = q 2^62
  unsigned long long Q = fix_mulhi(A, Y);
  if (Q >> 62) {
    ex++;
  } else {
    Q <<= 1;
  }
  // leading bit at 62: round at bit 9
  unsigned long long r = (Q + (1ull << 9)) >> 10;
  ex -= 1;
  if (r >> 53) {
    r >>= 1;
    ex++;
  }
  r = ((ua ^ ub) & (1ull << 63)) | ((unsigned long long)ex << 52) | (r & 0xfffffffffffffull);
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)r);
#else
  double d;
  __builtin_memcpy(&d, &r, 8);
  return d;
#endif
}

__host__ __device__ __forceinline__ bool fix_finite(double a) {
#ifdef __CUDA_ARCH__
  return fix_exp((unsigned long long)__double_as_longlong(a)) != 0x7ff;
#else
  unsigned long long u;
  __builtin_memcpy(&u, &a, 8);
  return fix_exp(u) != 0x7ff;
#endif
}

}  // namespace gsls
