// swe_fp64.cuh -- correctly rounded FP64 division and square root on the
// integer pipe.
//
// On GB300 the FP64 pipe retires 2 lanes per SM per cycle (measured 1.26
// TFLOP/s), so one warp-wide DFMA holds an SM partition's FP64 pipe for about
// 64 cycles, and a hardware division or square root is a chain of 7-10 of them.
// The integer pipe issues one warp instruction per cycle.  These routines
// compute IEEE round-to-nearest-even a / b and sqrt(x) from the 53-bit integer
// significands, with a single-precision estimate, one Newton step in 32-bit
// fixed point, two 31-bit digits and an exact remainder comparison, so the
// result equals the hardware instruction bit for bit.  Operands or results that
// are zero, subnormal, infinite or NaN take the hardware instruction.
#pragma once

#include <cuda_runtime.h>

namespace swe {

#if defined(__CUDACC__)

// Bit moves between a double and a 64-bit integer that the optimiser cannot
// see through.  With a plain reinterpretation, integer sign-mask operations on
// the bits (x & 0x7FF..F, x | sign, x ^ sign) are folded back into FP64 abs /
// negate instructions, which issue on the FP64 pipe (measured: an integer-key
// min of two doubles cost two FP64 instructions).
__device__ __forceinline__ long long dbits(double x) {
  long long r;
  asm("mov.b64 %0, %1;" : "=l"(r) : "d"(x));
  return r;
}
__device__ __forceinline__ double dfrom(long long r) {
  double x;
  asm("mov.b64 %0, %1;" : "=d"(x) : "l"(r));
  return x;
}

namespace fp64detail {

constexpr unsigned long long kM52 = (1ull << 52) - 1ull;
constexpr unsigned long long kHid = 1ull << 52;

__device__ __forceinline__ unsigned long long bits(double x) { return (unsigned long long)dbits(x); }
__device__ __forceinline__ double from_bits(unsigned long long u) { return dfrom((long long)u); }

// The hardware instructions for the rare operands, kept out of line so that
// the common path never issues them (predicated in-line copies would cost FP64
// pipe slots on every call).
static __device__ __noinline__ double ddiv_hw(double a, double b) { return __ddiv_rn(a, b); }
static __device__ __noinline__ double dsqrt_hw(double x) { return __dsqrt_rn(x); }

// 2^32 f for a float f in [0.5, 1), from its bits (an integer-to-float
// conversion would do, at eight times the issue cost)
__device__ __forceinline__ unsigned unit_fixed32(float f) { return (__float_as_uint(f) << 8) | 0x80000000u; }
// MUFU estimates (relative error about 2^-23), held inside [0.5, 1)
__device__ __forceinline__ unsigned rcp_seed(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return unit_fixed32(fmaxf(fminf(r, 0.99999994f), 0.5f));
}
__device__ __forceinline__ unsigned rsqrt_seed(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return unit_fixed32(fmaxf(fminf(r, 0.99999994f), 0.5f));
}

}  // namespace fp64detail

// 0.5 x and -x exactly, on the integer pipe: halving lowers the exponent by
// one; zeros, subnormals and the smallest normals (value M 2^-1074, M < 2^53)
// halve M with ties to even; infinities and NaNs are returned unchanged.
__device__ __forceinline__ double dhalf_rn(double x) {
  using namespace fp64detail;
  const unsigned long long u = bits(x);
  const unsigned e = (unsigned)(u >> 52) & 0x7FFu;
  if (e >= 2u && e != 0x7FFu) return from_bits(u - kHid);
  if (e == 0x7FFu) return x;
  const unsigned long long M = u & ((1ull << 53) - 1ull);
  const unsigned long long H = (M >> 1) + (M & (M >> 1) & 1ull);
  return from_bits((u & 0x8000000000000000ull) | H);
}
__device__ __forceinline__ double dneg(double x) {
  return fp64detail::from_bits(fp64detail::bits(x) ^ 0x8000000000000000ull);
}

// Method of ddiv_rn and dsqrt_rn.  Both keep every step within 32 x 32 -> 64
// bit products: a 32-bit reciprocal (square root) from the MUFU estimate and
// one Newton step (y' = y + y (1 - b y), y' = y + y (1 - x y^2) / 2), then the
// quotient (root) as two 31-bit digits with the running remainder held modulo
// 2^64 (it is far smaller than that), the second digit signed.  The digits
// leave an error of a few units 4 (5) bits below the last place, so the
// candidate m0 they give is within (-0.3, 1.3) of the true value in units of
// the last place, and one exact comparison with m0 + 1/2 rounds it.  (A tie
// cannot occur: a quotient or root of 53-bit significands never lies half way
// between two of them.)
//
// What bounds them is issue and, on small meshes, their own latency: a flux
// evaluation holds eight, and with the 128-bit Newton steps used before (about
// 290 instructions, 815 cycles each) the edge kernel issued 2536 instructions
// per warp for its 62 FP64 ones.  Measured, SSPRK2 step before -> now: 8192-cell
// Thacker bowl 172 -> 154 us, 1M-cell dam break 976 -> 945 us (k_flux 199 ->
// 187 us).  At this length they are inlined (out of line 0.5-1 % slower; the
// longer form was 5 % faster out of line).

// ma = significand of the dividend in [mb, 2 mb), mb = the divisor's in
// [2^52, 2^53): ma / mb rounded to 53 bits, in [2^52, 2^53].
__device__ __forceinline__ unsigned long long div_significand(unsigned long long ma, unsigned long long mb) {
  using namespace fp64detail;
  const unsigned d = (unsigned)(mb >> 21);  // top 32 bits
  const unsigned r0 = rcp_seed(__uint_as_float(0x3F800000u | ((d >> 8) & 0x7FFFFFu)));
  // R = 2^84 / mb to 2 units: |e| < 2^42
  const long long e = (long long)(0x8000000000000000ull - (unsigned long long)d * r0);
  const unsigned R = r0 + (unsigned)(__mulhi((int)(e >> 12), (int)(r0 >> 1)) >> 18);
  // ma / mb = (q1 + q2 2^-26) 2^-30 + rem2 / (mb 2^56)
  const unsigned q1 = __umulhi((unsigned)(ma >> 22), R);
  const long long rem1 = (long long)((ma << 30) - (unsigned long long)q1 * mb);  // within 6 mb < 2^56
  const int q2 = __mulhi((int)(rem1 >> 25), (int)(R >> 1));
  const long long rem2 = (long long)(((unsigned long long)rem1 << 26) - (unsigned long long)(long long)q2 * mb);
  const unsigned long long Q = ((unsigned long long)q1 << 26) + (unsigned long long)(long long)q2;
  const long long part = (long long)((Q & 15ull) * mb) + rem2;  // 16 (true - m0) mb
  return (Q >> 4) + (part > (long long)(mb << 3) ? 1ull : 0ull);
}

// M in [2^52, 2^54): sqrt(M 2^52) rounded to an integer in [2^52, 2^53].
__device__ __forceinline__ unsigned long long sqrt_significand(unsigned long long M) {
  using namespace fp64detail;
  const unsigned X = (unsigned)(M >> 22);  // x = X 2^-30 in [1, 4)
  const float f = (X >> 31) ? __uint_as_float(0x40000000u | ((X >> 8) & 0x7FFFFFu))
                            : __uint_as_float(0x3F800000u | ((X >> 7) & 0x7FFFFFu));
  const unsigned r0 = rsqrt_seed(f);
  // R = 2^32 / sqrt(x) to 3 units: |e| < 2^42
  const long long e = (long long)(0x4000000000000000ull - (unsigned long long)X * __umulhi(r0, r0));
  const unsigned R = r0 + (unsigned)(__mulhi((int)(e >> 11), (int)(r0 >> 1)) >> 19);
  // sqrt(M) = (s1 + s2 2^-27) 2^-4 to a few units of 2^-31
  const unsigned s1 = __umulhi(X, R);
  const long long rem1 = (long long)((M << 8) - (unsigned long long)s1 * s1);  // within 4 * 2 s1 < 2^34
  const int s2 = __mulhi((int)(rem1 >> 3), (int)(R >> 1));
  const unsigned long long S = ((unsigned long long)s1 << 27) + (unsigned long long)(long long)s2;
  const unsigned long long m0 = S >> 5;
  const long long rem = (long long)((M << 52) - m0 * m0);  // (true - m0)(true + m0), modulo 2^64
  return m0 + (rem > (long long)m0 ? 1ull : 0ull);
}

static __device__ __forceinline__ double ddiv_rn(double a, double b) {
  using namespace fp64detail;
  const unsigned long long ua = bits(a), ub = bits(b);
  const unsigned ea = (unsigned)(ua >> 52) & 0x7FFu, eb = (unsigned)(ub >> 52) & 0x7FFu;
  if (ea - 1u >= 2046u || eb - 1u >= 2046u) {
    // +-0 / normal (still water: zero momentum over a depth) stays in line
    if ((ua << 1) == 0ull && eb - 1u < 2046u) return from_bits((ua ^ ub) & 0x8000000000000000ull);
    return ddiv_hw(a, b);
  }
  unsigned long long ma = (ua & kM52) | kHid;
  const unsigned long long mb = (ub & kM52) | kHid;
  int E = (int)ea - (int)eb + 1023;
  if (ma < mb) {
    ma <<= 1;
    --E;
  }
  if (E < 1 || E > 2046) return ddiv_hw(a, b);
  // a significand of 2^53 carries into the exponent (and 2046 + 1 is infinity)
  return from_bits(((ua ^ ub) & 0x8000000000000000ull) |
                   (((unsigned long long)(unsigned)(E - 1) << 52) + div_significand(ma, mb)));
}

static __device__ __forceinline__ double dsqrt_rn(double x) {
  using namespace fp64detail;
  const unsigned long long ux = bits(x);
  const unsigned ex = (unsigned)(ux >> 52) & 0x7FFu;
  if (ex - 1u >= 2046u || (ux >> 63)) return (ux << 1) == 0ull ? x : dsqrt_hw(x);  // sqrt(+-0) = +-0 (dry side)
  // x = M 2^(e - 52) with an even e; 1023 is odd, so an even biased exponent is an odd e
  unsigned long long M = (ux & kM52) | kHid;
  if (!(ex & 1u)) M <<= 1;
  return from_bits(((unsigned long long)((ex + 1u) / 2u + 510u) << 52) + sqrt_significand(M));
}

// a b rounded to nearest even, on the integer pipe: the 106-bit product of the
// significands in four 32 x 32 -> 64 multiply-adds, shifted by 11 or 12 and
// rounded through the carry of the remainder.  For zeros and for exponents that
// keep the product normal (2^-511 to 2^511 each); anything else sets *other and
// the caller redoes its whole evaluation with the FP64 instructions.  (A
// fallback multiplication here, even never taken, is issued predicated off and
// takes its FP64 slot: 20 of the edge flux's 49.)  26 instructions, 22 of them
// on the ALU; the order of the words below is what gets them there.
__device__ __forceinline__ double dmul_rn(double a, double b, bool* other) {
  using namespace fp64detail;
  const unsigned long long ua = bits(a), ub = bits(b);
  const unsigned al = (unsigned)ua, ah = (unsigned)(ua >> 32), bl = (unsigned)ub, bh = (unsigned)(ub >> 32);
  const unsigned ma = (ah & 0xFFFFFu) | 0x100000u, mb = (bh & 0xFFFFFu) | 0x100000u;
  const unsigned long long p0 = (unsigned long long)al * bl;
  const unsigned long long p1 = (unsigned long long)al * mb + ((unsigned long long)ma * bl + (p0 >> 32));
  const unsigned long long p2 = (unsigned long long)ma * mb + (p1 >> 32);
  const unsigned top = (unsigned)(p2 >> 41);  // 1: the product is in [2, 4)
  const unsigned sh = 12u - top;
  unsigned hi = __funnelshift_l((unsigned)p2, (unsigned)(p2 >> 32), sh);
  unsigned lo = __funnelshift_l((unsigned)p1, (unsigned)p2, sh);
  const unsigned rem = ((unsigned)p1 << sh) | (min((unsigned)p0, 1u) | (lo & 1u));
  // sign and exponent: (ah - ma) + (bh - mb) adds the biased exponents less two
  // and, modulo 2^32, the signs; the hidden bit of hi adds one to the exponent
  const unsigned e = (ah - ma) + (bh - mb) + (top << 20) - (1022u << 20);
  unsigned t;
  asm("add.cc.u32 %0, %3, 0x7FFFFFFF;\n\t"  // carry: rem > half
      "addc.cc.u32 %1, %1, 0;\n\t"
      "addc.u32 %2, %2, %4;"
      : "=r"(t), "+r"(lo), "+r"(hi)
      : "r"(rem), "r"(e));
  // exponents outside [512, 1534]
  if ((ah << 1) - (512u << 21) >= (1023u << 21) || (bh << 1) - (512u << 21) >= (1023u << 21)) {
    const bool za = (ua << 1) == 0ull, zb = (ub << 1) == 0ull;
    if (!((za && (bh << 1) < 0xFFE00000u) || (zb && (ah << 1) < 0xFFE00000u))) *other = true;
    lo = 0u;
    hi = (ah ^ bh) & 0x80000000u;
  }
  return from_bits(((unsigned long long)hi << 32) | lo);
}

#endif  // __CUDACC__

}  // namespace swe
