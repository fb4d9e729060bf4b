// swe_physics.cuh -- point-wise physics of the SWE_FVM step, shared by the
// host-side geometry precompute and the sm_103a kernels.
//
// Every function restates one piece of the reference (NikitaMatckevich/
// SWE_FVM) with the same operation order, so that the device results match
// the CPU restatement bit for bit when the kernels are built without FMA
// contraction.  g = 1 throughout (the reference is nondimensional).
#pragma once

#include <cmath>
#include <cstdint>

#include "swe_fp64.cuh"

#if defined(__CUDACC__)
#define SWE_HD __host__ __device__ __forceinline__
#else
#define SWE_HD inline
#endif

namespace swe {

// Division and square root: the exact integer-pipe routines on the device
// (bit-identical to IEEE a / b and sqrt), the IEEE operators on the host.
#if defined(__CUDA_ARCH__)
#define SWE_DIV(a, b) ::swe::ddiv_rn((a), (b))
#define SWE_SQRT(x) ::swe::dsqrt_rn((x))
#else
#define SWE_DIV(a, b) ((a) / (b))
#define SWE_SQRT(x) std::sqrt((x))
#endif
// 0.5 x and -x (exact operations; on the device without FP64 instructions)
#if defined(__CUDA_ARCH__)
#define SWE_HALF(x) ::swe::dhalf_rn((x))
#define SWE_NEG(x) ::swe::dneg((x))
#else
#define SWE_HALF(x) (0.5 * (x))
#define SWE_NEG(x) (-(x))
#endif

// include/Includes.h:30
constexpr double kTol = 1e-13;
// include/Bathymetry.h:5-8
constexpr double kWetDepth = 1e-12;
// include/Fluxes.h:28,37,73
constexpr double kMinCapture = 1e-10;
// include/Assigners.h:30-32
constexpr double kEta1 = 1e-3;
constexpr double kEta2 = 1e-6;
constexpr double kEta4 = 1e-12;
constexpr double kSqrt2 = 1.4142135623730951;  // std::sqrt(2), correctly rounded

// ------------------------------------------------------------ comparisons
// On GB300 a warp-wide FP64 instruction, compares included, occupies the
// FP64 pipe for ~64 cycles, while the integer pipe issues one per cycle.  On the
// device every comparison therefore goes through integer keys: for non-NaN
// doubles, key(x) = (bits < 0) ? -(bits & 0x7FF..F) : bits is monotone and maps
// -0 and +0 to the same key, so a < b <=> key(a) < key(b) exactly.  (A NaN
// anywhere makes the state non-finite, which the update kernel reports.)  The
// host keeps the IEEE comparisons: the two agree on every non-NaN input.
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ long long fkey(double x) {
  const long long i = dbits(x);
  return i < 0 ? -(i & 0x7FFFFFFFFFFFFFFFll) : i;
}
__device__ __forceinline__ long long fbits(double x) { return dbits(x); }
SWE_HD bool dlt(double a, double b) { return fkey(a) < fkey(b); }
SWE_HD bool dle(double a, double b) { return fkey(a) <= fkey(b); }
// x > c and x < c for a constant c > 0: the signed bit patterns order them
SWE_HD bool dgtc(double x, double c) { return fbits(x) > fbits(c); }
SWE_HD bool dltc(double x, double c) { return fbits(x) < fbits(c); }
// x > 0 and x >= 0
SWE_HD bool dgt0(double x) { return fbits(x) > 0; }
SWE_HD bool dge0(double x) { return fkey(x) >= 0; }
#else
SWE_HD bool dlt(double a, double b) { return a < b; }
SWE_HD bool dle(double a, double b) { return a <= b; }
SWE_HD bool dgtc(double x, double c) { return x > c; }
SWE_HD bool dltc(double x, double c) { return x < c; }
SWE_HD bool dgt0(double x) { return x > 0.; }
SWE_HD bool dge0(double x) { return x >= 0.; }
#endif

SWE_HD bool is_wet(double h) { return dgtc(h, kWetDepth); }
// std::min / std::max (first argument kept on ties)
SWE_HD double smin(double a, double b) { return dlt(b, a) ? b : a; }
SWE_HD double smax(double a, double b) { return dlt(a, b) ? b : a; }

// ---------------------------------------------------------------- geometry
// src/PointOperations.cpp:42-48: slope (gx, gy) of the plane through three
// points, 2x2 partial-pivot LU (pivot: first row with the largest |a_i0|).
SWE_HD void plane_gradient(double p0x, double p0y, double p0z, double p1x, double p1y, double p1z, double p2x,
                           double p2y, double p2z, double* gx, double* gy) {
  double a00 = p1x - p0x, a01 = p1y - p0y, b0 = p1z - p0z;
  double a10 = p2x - p0x, a11 = p2y - p0y, b1 = p2z - p0z;
  if (dlt(fabs(a00), fabs(a10))) {
    double t;
    t = a00; a00 = a10; a10 = t;
    t = a01; a01 = a11; a11 = t;
    t = b0; b0 = b1; b1 = t;
  }
  double l10 = a10;
  if (a00 != 0.) l10 = SWE_DIV(a10, a00);
  double u11 = a11 - l10 * a01;
  double y1 = b1 - l10 * b0;
  double x1 = SWE_DIV(y1, u11);
  double x0 = SWE_DIV(b0 - a01 * x1, a00);
  *gx = x0;
  *gy = x1;
}

// Bit patterns on the host and the device.
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ unsigned long long ubits(double x) { return (unsigned long long)dbits(x); }
__device__ __forceinline__ double ufrom(unsigned long long u) { return dfrom((long long)u); }
#else
SWE_HD unsigned long long ubits(double x) {
  union { double d; unsigned long long u; } c;
  c.d = x;
  return c.u;
}
SWE_HD double ufrom(unsigned long long u) {
  union { double d; unsigned long long u; } c;
  c.u = u;
  return c.d;
}
#endif
// a / b in single precision where only a correction or a starting point depends on it
SWE_HD float quick_div(float a, float b) {
#if defined(__CUDA_ARCH__)
  return __fdividef(a, b);
#else
  return a / b;
#endif
}
SWE_HD bool negative(double x) { return (ubits(x) >> 63) != 0ull; }
SWE_HD double magnitude(double x) { return ufrom(ubits(x) & 0x7FFFFFFFFFFFFFFFull); }

// (int)log2(x) for finite x > 0, truncated toward zero, from the exponent bits
// (src/PointOperations.cpp:33).
SWE_HD int trunc_log2(double x) {
  const unsigned long long u = ubits(x);
  int e = (int)(u >> 52) - 1022;  // x = m 2^e, m in [0.5, 1)
  bool half = (u << 12) == 0ull;
  if ((u >> 52) == 0ull) half = frexp(x, &e) == 0.5;  // subnormal
  if (half) return e - 1;
  return (e >= 1) ? e - 1 : e;
}

// Correctly rounded cube root (round to nearest, ties to even) for the
// PartWet1 level (src/MUSCLObject.cpp:103).  The math libraries' cbrt are
// faithful, not correctly rounded, and the CUDA and host ones differ in the
// last bit; this one is exact on both.  Method: x = Mx 2^E with a 53-bit
// integer Mx; N = Mx 2^t with t in {107, 108, 109} chosen so that 3 | (E - t)
// and N in [2^159, 2^162); Y = floor(cbrt(N)) in [2^53, 2^54) is found from an
// estimate corrected with exact 192-bit integer cubes; its lowest bit and the
// remainder N - Y^3 round it to 53 bits.  The estimate is a single-precision
// root and two Newton steps whose corrections are single-precision quotients
// (2^-22 -> 2^-44 -> a few units): a library root, frexp and ldexp in its place
// put some four thousand cycles on the chain of every thin cell.
struct U192 {
  unsigned long long w[3];  // little-endian limbs
};
SWE_HD U192 u192_cube(unsigned long long y) {
  // y < 2^55: y^2 < 2^110 fits 128 bits, y^3 < 2^165 fits 192 bits
  unsigned __int128 y2 = (unsigned __int128)y * y;
  unsigned __int128 lo = (unsigned __int128)(unsigned long long)y2 * y;
  unsigned __int128 hi = (unsigned __int128)(unsigned long long)(y2 >> 64) * y;
  U192 r;
  r.w[0] = (unsigned long long)lo;
  unsigned __int128 mid = (lo >> 64) + (unsigned long long)hi;
  r.w[1] = (unsigned long long)mid;
  r.w[2] = (unsigned long long)((mid >> 64) + (hi >> 64));
  return r;
}
// a <= b
SWE_HD bool u192_le(const U192& a, const U192& b) {
  if (a.w[2] != b.w[2]) return a.w[2] < b.w[2];
  if (a.w[1] != b.w[1]) return a.w[1] < b.w[1];
  return a.w[0] <= b.w[0];
}
SWE_HD double cbrt_rn(double x) {
  if (!(x == x) || x == 0. || (ubits(x) << 1) == (0x7FFull << 53)) return x + x;  // NaN, +-0, +-inf
  const bool neg = negative(x);
  double ax = magnitude(x);
  int scale = 0;
  if (ax < 2.2250738585072014e-308) {  // subnormal: scale by 2^54
    ax = ax * 18014398509481984.0;
    scale = -18;
  }
  const unsigned long long ua = ubits(ax);
  const unsigned long long Mx = (ua & ((1ull << 52) - 1ull)) | (1ull << 52);
  const int E = (int)(ua >> 52) - 1075;  // ax = Mx 2^E
  const int k = ((E - 107) % 3 + 3) % 3;  // t = 107 + k
  // N = Mx 2^t as 192 bits (t - 64 in {43, 44, 45})
  U192 N;
  N.w[0] = 0ull;
  N.w[1] = Mx << (43 + k);
  N.w[2] = Mx >> (21 - k);
  // u = Mx 2^(k - 52) in [1, 8), exactly; c -> cbrt(u) = cbrt(N) 2^-53
  const double u = ufrom((Mx & ((1ull << 52) - 1ull)) | ((unsigned long long)(1023 + k) << 52));
  double c = (double)cbrtf((float)u);
  c -= (double)quick_div((float)(c * c * c - u), (float)(3. * c * c));
  {
    const double p = c * c, e = fma(c, c, -p);
    const double r = fma(p, c, -u) + e * c;  // c^3 - u
    c -= (double)quick_div((float)r, (float)(3. * p));
  }
  const double est = c * 9007199254740992.0;  // 2^53
  unsigned long long Y = est >= 18014398509481983.0 ? (1ull << 54) - 1 : (unsigned long long)est;
  if (Y < (1ull << 53)) Y = 1ull << 53;
  U192 q = u192_cube(Y);
  for (int it = 0; it < 64 && !u192_le(q, N); ++it) q = u192_cube(--Y);
  for (int it = 0; it < 64; ++it) {
    const U192 q1 = u192_cube(Y + 1);
    if (!u192_le(q1, N)) break;
    ++Y;
    q = q1;
  }
  const bool sticky = q.w[0] != N.w[0] || q.w[1] != N.w[1] || q.w[2] != N.w[2];
  unsigned long long R = Y >> 1;  // in [2^52, 2^53)
  if ((Y & 1ull) && (sticky || (R & 1ull))) ++R;
  // R 2^s with s = (E - t) / 3 + 1 + scale: the result is normal, a carry of R
  // to 2^53 goes into the exponent
  const int s = (E - 107 - k) / 3 + 1 + scale;
  const double r = ufrom(((unsigned long long)(s + 1074) << 52) + R);
  return neg ? -r : r;
}

// include/CubicPolyMath.h:13-15: x^3 + b x^2 + c x + d
SWE_HD double cubic(double d, double c, double b, double x) { return x * x * x + b * x * x + c * x + d; }

// |a| > |b| for two magnitudes, from their bits
SWE_HD bool above(double x, double bound) { return ubits(x) > ubits(bound); }

// The reference's bisection (src/PointOperations.cpp:26-40), bit for bit.  Its
// result is the last midpoint of a path that only the sign of the computed f
// at each midpoint decides, and away from the root that sign is known without
// evaluating f.  Let E bound the error of a computed value anywhere on the
// interval, let f have one curvature there, and let lo < hi be points where the
// computed |f| exceeds 2 E (as at the ends of the interval) with the signs of
// f(xmin) and f(xmax).  Then the true |f| exceeds E on all of [xmin, lo] and
// [hi, xmax]: the side on which f runs away from zero is monotone, and on the
// other a convex (concave) f lies on the far side of the chord between two such
// points.  (Where lo <= xmin or hi >= xmax that part is empty.)  So f is
// evaluated only between lo and hi, some units of rounding apart: 7 to 20 of
// the 51 evaluations, each 5 to 8 FP64 operations of 64 cycles for the warp.
// lo and hi come from a single-precision bisection and two Newton steps; where
// the check fails the whole path is walked.  With cbrt_rn above, SSPRK2 pass
// before -> now: 8192-cell Thacker bowl 154 -> 132 us a step, 250k-cell coast
// 504 -> 436 us (k_recon1 86 -> 57 us, k_recon2 47 -> 43 us).
// The float root s in [0, 1] of ((p3 s + p2) s + p1) s + p0, whose value at 0
// has the sign neg: 20 halvings.
SWE_HD float unit_root(float p3, float p2, float p1, float p0, bool neg) {
  float s = 0.f, w = 0.5f;
  for (int it = 0; it < 20; ++it) {
    const float sm = s + w;
    const float f = ((p3 * sm + p2) * sm + p1) * sm + p0;
    if ((f < 0.f) == neg) s = sm;
    w *= 0.5f;
  }
  return s + w;
}

// (xmin + xmax) / 2 rounded as the reference's 0.5 (xmin + xmax).
SWE_HD double midpoint(double xmin, double xmax) {
  const unsigned long long A = ubits(xmin), Z = ubits(xmax);
  const unsigned ex = (unsigned)(A >> 52);
  if (ex == (unsigned)(Z >> 52) && (ex & 0x7FFu) > 2u && (ex & 0x7FFu) < 0x7FEu) {
    // one sign and binade: the mean of the bit patterns, rounded to even
    const unsigned long long h = (A & Z) + ((A ^ Z) >> 1);
    return ufrom(h + (h & (A ^ Z) & 1ull));
  }
  return SWE_HALF(xmin + xmax);
}

// Where the computed sign of f must be looked at: outside [lo, hi] it is that of
// the nearer end.
struct Bracket {
  double lo, hi;
};

// Lower and upper bounds lo <= root <= hi as above for x^3 + c x + d on [0, 1]
// (convex) with the ends' computed values fmin and fmax of opposite signs.
// two: how the two points' computed values are had (a lane group evaluates them
// together, with collectives: no path around the call).
template <class Two>
SWE_HD Bracket bracket01(double d, double c, double fmin_, double fmax_, Two&& two) {
  const bool neg_min = negative(fmin_);
  Bracket r{0., 1.};
  // |computed f - f| <= u (5 x^3 + 3 |c| x + |d|), held a little larger
  const double E = 6e-16 + 3.6e-16 * magnitude(c) + 1.3e-16 * magnitude(d);
  const float g = quick_div(1.0f, fmaxf(fabsf((float)fmin_), fabsf((float)fmax_)));
  double x = (double)unit_root(g, 0.f, (float)c * g, (float)fmin_ * g, neg_min);
  double slope = 0.;
  for (int q = 0; q < 2; ++q) {
    const double y = fma(x, x, c);
    slope = fma(2. * x, x, y);
    x -= (double)quick_div((float)fma(y, x, d), (float)slope);
  }
  const double gap = (double)quick_div((float)(2.6 * E), fabsf((float)slope)) + 4.5e-16;
  const double l = x - gap, h = x + gap, E2 = 2. * E;
  double fl, fh;
  two(l, h, &fl, &fh);
  const bool at0 = !dlt(0., l), at1 = !dlt(h, 1.);
  const bool ok = (at0 || (negative(fl) == neg_min && above(magnitude(fl), E2) && above(magnitude(fmin_), E2))) &&
                  (at1 || (negative(fh) != neg_min && above(magnitude(fh), E2) && above(magnitude(fmax_), E2))) &&
                  dlt(l, 1.) && dlt(0., h) && above(1e280, E) && x == x;
  if (ok && !at0) r.lo = l;
  if (ok && !at1) r.hi = h;
  return r;
}

// The bisection of [0, 1] has dyadic midpoints, so its steps down to the last
// interval that holds [r.lo, r.hi] are taken at once: their number (at most
// most), and that interval.
SWE_HD int dyadic_steps(const Bracket& r, int most, double* xmin, double* xmax) {
  // floor(lo 2^62) and ceil(hi 2^62) - 1: their common leading bits are steps
  const unsigned long long ul = ubits(r.lo), uh = ubits(r.hi);
  const int sl = 1013 - (int)(ul >> 52), sh = 1013 - (int)(uh >> 52);
  const unsigned long long hid = 1ull << 52, ml = (ul & (hid - 1)) | hid, mh = (uh & (hid - 1)) | hid;
  unsigned long long fl = 0ull, fh = (1ull << 62) - 1ull;
  if (ul != 0ull) fl = sl <= 0 ? ml << -sl : sl < 64 ? ml >> sl : 0ull;
  if (uh != ubits(1.)) fh = sh <= 0 ? (mh << -sh) - 1ull : sh < 53 ? (mh - 1ull) >> sh : 0ull;
  const unsigned long long diff = fl ^ fh;
  int k = 0;
  for (int w = 32; w > 0; w >>= 1)
    if (k + w <= 62 && (diff >> (62 - k - w)) == 0ull) k += w;
  if (k > most) k = most;
  const unsigned long long j = fl >> (62 - k);
  const double scale = ufrom((unsigned long long)(1023 - k) << 52);  // 2^-k
  *xmin = (double)j * scale;
  *xmax = (double)(j + 1ull) * scale;
  return k;
}

// The bracket for x^3 + b x^2 + c x + d on [xmin, xmax], of width w.
template <class Two>
SWE_HD Bracket bracket(double d, double c, double b, double xmin, double xmax, double w, double fmin_, double fmax_,
                       Two&& two) {
  const bool neg_min = negative(fmin_);
  Bracket r{xmin, xmax};
  // f'' / 2 at the ends, rounded twice (PartWet1's is -3 b13 + 3 b13 at the upper
  // one: a last bit of b there bends f by less than E)
  const double c0 = 3. * xmin + b, c1 = 3. * xmax + b;
  const bool curved = (dle(0., c0) && dle(0., c1)) || (dle(c0, 0.) && dle(c1, 0.));
  // f(xmin + w s) / |f| in single precision, s in [0, 1]
  const float fw = (float)w, fc0 = (float)c0;
  const float g = quick_div(1.0f, fmaxf(fabsf((float)fmin_), fabsf((float)fmax_)));
  const double s0 = fma(xmin, c0 + b, c);  // f'(xmin)
  const float p1 = (float)s0 * fw * g, p2 = fc0 * fw * fw * g, p3 = fw * fw * fw * g;
  double x = fma(w, (double)unit_root(p3, p2, p1, (float)fmin_ * g, neg_min), xmin);
  double slope = 0.;
  for (int q = 0; q < 2; ++q) {
    const double y = x + b, z = fma(x, y, c);
    slope = fma(x, y + x, z);
    x -= (double)quick_div((float)fma(z, x, d), (float)slope);
  }
  // |computed f - f| <= u (5 |x|^3 + 5 |b| x^2 + 3 |c| |x| + |d|), a little larger
  const double m = smax(magnitude(xmin), magnitude(xmax));
  const double E = fma(6e-16, fma(m + magnitude(b), m, magnitude(c)) * m, 1.3e-16 * magnitude(d));
  const double gap = fma(4.5e-16, m, (double)quick_div((float)(2.6 * E), fabsf((float)slope)));
  const double l = x - gap, h = x + gap, E2 = 2. * E;
  double fl, fh;
  two(l, h, &fl, &fh);
  const bool at0 = !dlt(xmin, l), at1 = !dlt(h, xmax);
  const bool ok = (at0 || (negative(fl) == neg_min && above(magnitude(fl), E2) && above(magnitude(fmin_), E2))) &&
                  (at1 || (negative(fh) != neg_min && above(magnitude(fh), E2) && above(magnitude(fmax_), E2))) &&
                  dlt(l, xmax) && dlt(xmin, h) && above(E, 1e-280) && above(1e280, E) && x == x && curved;
  if (ok && !at0) r.lo = l;
  if (ok && !at1) r.hi = h;
  return r;
}

// x^3 + c x + d on [0, 1] (PartWet2).  The quadratic term is 0 x x, whose
// addition changes no bit of x^3 >= 0; f(0) is 0 + d and f(1) (1 + c) + d.
SWE_HD double cubic01(double d, double c, double x) { return x * x * x + c * x + d; }
SWE_HD double bisection01(double d, double c) {
  const double fmin_ = 0. + d, fmax_ = (1. + c) + d;
  const bool neg_min = negative(fmin_);
  if (neg_min == negative(fmax_)) return dlt(magnitude(fmin_), magnitude(fmax_)) ? 0. : 1.;
  const Bracket r = bracket01(d, c, fmin_, fmax_, [&](double l, double h, double* fl, double* fh) {
    *fl = cubic01(d, c, l);
    *fh = cubic01(d, c, h);
  });
  double xmin, xmax, x = 0.;
  for (int it = dyadic_steps(r, 50, &xmin, &xmax); it <= 50; it++) {
    x = midpoint(xmin, xmax);
    bool left;
    if (dle(x, r.lo)) left = true;
    else if (dle(r.hi, x)) left = false;
    else left = negative(cubic01(d, c, x)) == neg_min;
    if (left) xmin = x;
    else xmax = x;
  }
  return x;
}

// The general form.
SWE_HD double bisection(double d, double c, double b, double xmin, double xmax) {
  if ((ubits(b) | ubits(xmin)) == 0ull && ubits(xmax) == ubits(1.)) return bisection01(d, c);
  const double fmin_ = cubic(d, c, b, xmin);
  const double fmax_ = cubic(d, c, b, xmax);
  const bool neg_min = negative(fmin_);
  if (neg_min == negative(fmax_)) return dlt(magnitude(fmin_), magnitude(fmax_)) ? xmin : xmax;
  const double w = xmax - xmin;
  const int n = 50 + trunc_log2(w);
  Bracket r{xmin, xmax};
  if (n > 8)
    r = bracket(d, c, b, xmin, xmax, w, fmin_, fmax_, [&](double l, double h, double* fl, double* fh) {
      *fl = cubic(d, c, b, l);
      *fh = cubic(d, c, b, h);
    });
  double x = 0.;
  for (int it = 0; it <= n; it++) {
    x = midpoint(xmin, xmax);
    bool left;
    if (dle(x, r.lo)) left = true;
    else if (dle(r.hi, x)) left = false;
    else left = negative(cubic(d, c, b, x)) == neg_min;
    if (left) xmin = x;
    else xmax = x;
  }
  return x;
}

#if defined(__CUDACC__)
// The same by groups of 8 lanes, four bisections a warp.  Every lane of the warp
// calls together, the lanes of a group with the same operands, and the groups
// that have none with active = false.  The steps that the bracket decides are
// taken by comparison; then lane q > 0 of a group takes node q of the tree of
// the next seven midpoints, so that a round settles three steps for one
// evaluation.  All collectives are over the warp: with groups that run apart the
// FP64 pipe would issue each group's operations by themselves (64 cycles each).
template <bool UNIT>
__device__ double bisection_group(double d, double c, double b, double xmin, double xmax, bool active) {
  constexpr unsigned kWarp = 0xFFFFFFFFu;
  const int q = threadIdx.x & 7;
  auto f = [&](double x) { return UNIT ? cubic01(d, c, x) : cubic(d, c, b, x); };
  // the computed values at two points, one in the even lanes and one in the odd
  auto two = [&](double l, double h, double* fl, double* fh) {
    const double v = f((q & 1) ? h : l);
    *fl = __shfl_sync(kWarp, v, 0, 8);
    *fh = __shfl_sync(kWarp, v, 1, 8);
  };
  double fmin_, fmax_;
  if (UNIT) {
    fmin_ = 0. + d;
    fmax_ = (1. + c) + d;
  } else {
    two(xmin, xmax, &fmin_, &fmax_);
  }
  const bool neg_min = negative(fmin_);
  const bool same = neg_min == negative(fmax_);
  double x = same ? (dlt(magnitude(fmin_), magnitude(fmax_)) ? xmin : xmax) : 0.;
  int n = 50, it = 0;
  Bracket r;
  if (UNIT) {
    r = bracket01(d, c, fmin_, fmax_, two);
    it = dyadic_steps(r, n, &xmin, &xmax);
  } else {
    const double w = xmax - xmin;
    n = 50 + trunc_log2(w);
    const Bracket found = bracket(d, c, b, xmin, xmax, w, fmin_, fmax_, two);
    r = n > 8 ? found : Bracket{xmin, xmax};
  }
  if (same || !active) n = -1;
  // steps that the bracket decides
  auto key = [](double y) {  // ordered as the doubles are
    const long long u = (long long)ubits(y);
    return u < 0 ? -(u & 0x7FFFFFFFFFFFFFFFll) : u;
  };
  const long long klo = key(r.lo), khi = key(r.hi);
  bool plain = it <= n;
  while (__any_sync(kWarp, plain)) {
    if (plain) {
      const double mid = midpoint(xmin, xmax);
      const long long k = key(mid);
      if (k <= klo) xmin = x = mid;
      else if (khi <= k) xmax = x = mid;
      else plain = false;
      if (plain) plain = ++it <= n;
    }
  }
  const int node = q > 0 ? q : 1, depth = node > 3 ? 2 : node > 1 ? 1 : 0;
  while (__any_sync(kWarp, it <= n)) {
    // this lane's midpoint: down from the root by its node number's bits
    double a = xmin, z = xmax, mid = midpoint(a, z);
#pragma unroll
    for (int t = 0; t < 2; ++t)
      if (t < depth) {
        if ((node >> (depth - 1 - t)) & 1) a = mid;
        else z = mid;
        mid = midpoint(a, z);
      }
    const long long k = key(mid);
    const bool neg = negative(f(mid));
    const bool right = k <= klo || (k < khi && neg == neg_min);  // the path goes on right of mid
    const unsigned went = __ballot_sync(kWarp, right) >> (threadIdx.x & 24);
    const int levels = min(3, n - it + 1);
    int at = 1;
    if (levels > 1) at = 2 * at + ((went >> at) & 1u);
    if (levels > 2) at = 2 * at + ((went >> at) & 1u);
    const double xn = __shfl_sync(kWarp, mid, at, 8);
    const double an = __shfl_sync(kWarp, right ? mid : a, at, 8);
    const double zn = __shfl_sync(kWarp, right ? z : mid, at, 8);
    if (it <= n) {
      x = xn;
      xmin = an;
      xmax = zn;
      it += levels;
    }
  }
  return x;
}
#endif

// --------------------------------------------------------------- assigners
// src/Assigners.cpp:8-20: PrimAssigner (edge writes)
SWE_HD void prim_assign(double b, double w, double u, double v, double* ow, double* ou, double* ov) {
  double h = w - b;
  if (!is_wet(h)) {
    *ow = b; *ou = 0.; *ov = 0.;
    return;
  }
  if (dltc(h, kEta1)) {
    double s = SWE_DIV(kSqrt2 * h, SWE_SQRT(h * h + kEta2));
    u *= s;
    v *= s;
  }
  *ow = w; *ou = u; *ov = v;
}

// src/Assigners.cpp:28-44: ConsAssigner (cell writes)
SWE_HD void cons_assign(double b, double h, double hu, double hv, double* ow, double* ou, double* ov) {
  if (!is_wet(h)) {
    *ow = b; *ou = 0.; *ov = 0.;
    return;
  }
  double ih;
  if (dltc(h, kEta1)) ih = SWE_DIV(kSqrt2 * h, SWE_SQRT(h * h * h * h + kEta4));
  else ih = SWE_DIV(1., h);
  *ow = h + b;
  *ou = hu * ih;
  *ov = hv * ih;
}

// -------------------------------------------------------------- edge flux
// How a flux or update multiplies: on the integer pipe (SOFT, the same bits;
// dmul_rn) or on the FP64 pipe.  other is set when an operand was outside
// dmul_rn's range: the evaluation is then to be done again with Products<false>.
template <bool SOFT>
struct Products {
  bool other = false;
  SWE_HD double mul(double a, double b) {
#if defined(__CUDA_ARCH__)
    if (SOFT) return dmul_rn(a, b, &other);
#endif
    return a * b;
  }
};

// include/SpaceDisc.h:4-18: F.n of U = (h, hu, hv), g = 1; hh = h h
template <class M>
SWE_HD void elem_flux_hh(M& m, double nx, double ny, double h, double hu, double hv, double hh, double* f) {
  f[0] = 0.; f[1] = 0.; f[2] = 0.;
  if (is_wet(h)) {
    double hveln = m.mul(hu, nx) + m.mul(hv, ny);
    f[0] = hveln;
    const double q = SWE_DIV(hveln, h);
    const double p = SWE_HALF(hh);  // (0.5 h) h: halving is exact on either side of the product
    f[1] = m.mul(q, hu) + m.mul(p, nx);
    f[2] = m.mul(q, hv) + m.mul(p, ny);
  }
}
SWE_HD void elem_flux(double nx, double ny, double h, double hu, double hv, double* f) {
  Products<false> m;
  elem_flux_hh(m, nx, ny, h, hu, hv, h * h, f);
}

// Wave-speed plugins (src/Fluxes.cpp:5-26).  speeds() returns the pair the
// reference's Array<2> holds.
// What a flux evaluation can leave for its reverse: the wave speeds'
// intermediates and u* (the discrete adjoint's recompute stores them, see
// swe_flux_adjoint.cuh).  NoTape records nothing and compiles away.
struct NoTape {
  SWE_HD void speeds(double, double, double, double, double, double) const {}
  SWE_HD void ustar(double) const {}
};
// Edge e's intermediates into t[k * E + e]: cl, cr, uRoe, cRoe, a0, a1, u*.
struct EdgeTape {
  double* t;
  int E, e;
  SWE_HD void speeds(double cl, double cr, double uRoe, double cRoe, double a0, double a1) const {
    t[e] = cl;
    t[E + e] = cr;
    t[2 * E + e] = uRoe;
    t[3 * E + e] = cRoe;
    t[4 * E + e] = a0;
    t[5 * E + e] = a1;
  }
  SWE_HD void ustar(double us) const { t[6 * E + e] = us; }
};

struct Rusanov {
  static constexpr int id = 0;
  template <class M, class T>
  SWE_HD static void speeds(M& m, double ul, double hl, double ur, double hr, double* a0, double* a1,
                            const T& tape) {
    double cl = SWE_SQRT(hl), cr = SWE_SQRT(hr);
    double ap = smax(fabs(ul) + cl, fabs(ur) + cr);
    *a0 = -ap;
    *a1 = ap;
    tape.speeds(cl, cr, 0., 0., *a0, *a1);
  }
  SWE_HD static void speeds(double ul, double hl, double ur, double hr, double* a0, double* a1) {
    Products<false> m;
    speeds(m, ul, hl, ur, hr, a0, a1, NoTape{});
  }
};
struct Davis {
  static constexpr int id = 1;
  template <class M, class T>
  SWE_HD static void speeds(M& m, double ul, double hl, double ur, double hr, double* a0, double* a1,
                            const T& tape) {
    double cl = SWE_SQRT(hl), cr = SWE_SQRT(hr);
    *a0 = smin(ul - cl, ur - cr);
    *a1 = smax(ul + cl, ur + cr);
    tape.speeds(cl, cr, 0., 0., *a0, *a1);
  }
  SWE_HD static void speeds(double ul, double hl, double ur, double hr, double* a0, double* a1) {
    Products<false> m;
    speeds(m, ul, hl, ur, hr, a0, a1, NoTape{});
  }
};
struct Einfeldt {
  static constexpr int id = 2;
  template <class M, class T>
  SWE_HD static void speeds(M& m, double ul, double hl, double ur, double hr, double* a0, double* a1,
                            const T& tape) {
    double cl = SWE_SQRT(hl), cr = SWE_SQRT(hr);
    double uRoe = SWE_DIV(m.mul(cl, ul) + m.mul(cl, ur), cl + cr);  // the reference's cl * ur
    double cRoe = SWE_SQRT(SWE_HALF(hl + hr));
    *a0 = smin(ul - cl, uRoe - cRoe);
    *a1 = smax(ur + cr, uRoe + cRoe);
    tape.speeds(cl, cr, uRoe, cRoe, *a0, *a1);
  }
  SWE_HD static void speeds(double ul, double hl, double ur, double hr, double* a0, double* a1) {
    Products<false> m;
    speeds(m, ul, hl, ur, hr, a0, a1, NoTape{});
  }
};

// Everything a flux plugin reads about one interior edge: the geometry of the
// edge seen from its owner ("from", include/Fluxes.h:20,62-63) and the two
// reconstructed interface states.
struct EdgeGeom {
  double nx, ny;  // Domain::Norm(e, from)
  double tx, ty;  // Domain::Tang(e, from)
  double b;       // edge-centre bathymetry
  double lmin;    // min(2 A_from / L, 2 A_to / L)
};
struct SideState {
  double w, u, v;  // interface primitive values (EdgeField slot)
};
struct DepthState {
  double h, u, v;  // the same with the depth w - b
};
SWE_HD DepthState depth_state(const SideState& s, double b) { return DepthState{s.w - b, s.u, s.v}; }

// |cor| + speed for a speed >= 0 (without an operation where cor is zero)
SWE_HD double plus_coriolis(double cor, double speed) {
  return (ubits(cor) << 1) == 0ull ? speed : fabs(cor) + speed;
}

// Whether reach / speed can lower a minimum whose double's upper word is cap
// (kNoCap: always).  The upper word over 2^20 is the logarithm to base 2 plus
// 1023, short of it by at most 0.0861, so a difference above cap by twice that
// settles it (for normal numbers): three integer operations for the quotient's
// sixty-five.  In a jittered mesh nearly every edge is settled.
constexpr int kNoCap = 0x7FFFFFFF;
SWE_HD bool may_lower(double reach, double speed, int cap) {
  const int r = (int)(ubits(reach) >> 32), s = (int)(ubits(speed) >> 32);
  constexpr int kMargin = (1023 << 20) - 180668;  // 0.1723 2^20
  return cap == kNoCap || r < (1 << 20) || r - s + kMargin <= cap;
}

// Fluxes::HLL<W> (include/Fluxes.h:14-54).  *lw receives the edge's
// length-to-wavespeed ratio, or is left alone when the edge does not update it
// or cannot lower the minimum that cap describes (may_lower).
template <class W>
struct HLL {
  static constexpr int id = 0;
  SWE_HD static void eval(const EdgeGeom& g, const SideState& L, const SideState& R, double cor, double* lw,
                          double* F) {
    Products<false> m;
    eval_depth(m, g, depth_state(L, g.b), depth_state(R, g.b), cor, kNoCap, lw, F, NoTape{});
  }
  template <class M, class T>
  SWE_HD static void eval_depth(M& m, const EdgeGeom& g, const DepthState& L, const DepthState& R, double cor,
                                int cap, double* lw, double* F, const T& tape) {
    const double hl = L.h, hr = R.h;
    double ul = m.mul(L.u, g.nx) + m.mul(L.v, g.ny);
    double ur = m.mul(R.u, g.nx) + m.mul(R.v, g.ny);
    F[0] = 0.; F[1] = 0.; F[2] = 0.;
    if (!dgtc(hl + hr, kMinCapture)) return;
    double a0, a1;
    W::speeds(m, ul, hl, ur, hr, &a0, &a1, tape);
    double al = smin(0., a0);
    double ar = smax(0., a1);
    if (!dgtc(ar - al, kMinCapture)) return;
    const double speed = plus_coriolis(cor, smax(-al, ar));
    if (may_lower(g.lmin, speed, cap)) *lw = SWE_DIV(g.lmin, speed);
    double Ul[3] = {hl, m.mul(hl, L.u), m.mul(hl, L.v)};
    double Ur[3] = {hr, m.mul(hr, R.u), m.mul(hr, R.v)};
    double Fl[3], Fr[3];
    elem_flux_hh(m, g.nx, g.ny, Ul[0], Ul[1], Ul[2], m.mul(hl, hl), Fl);
    elem_flux_hh(m, g.nx, g.ny, Ur[0], Ur[1], Ur[2], m.mul(hr, hr), Fr);
    const double aa = al * ar, d = ar - al;
#pragma unroll
    for (int q = 0; q < 3; ++q)
      F[q] = SWE_DIV(m.mul(ar, Fl[q]) - m.mul(al, Fr[q]) +
                         m.mul(aa, Ur[q] - Ul[q]), d);
  }
};

// Fluxes::HLLC<W> (include/Fluxes.h:56-111)
template <class W>
struct HLLC {
  static constexpr int id = 1;
  SWE_HD static void eval(const EdgeGeom& g, const SideState& L, const SideState& R, double cor, double* lw,
                          double* F) {
    Products<false> m;
    eval_depth(m, g, depth_state(L, g.b), depth_state(R, g.b), cor, kNoCap, lw, F, NoTape{});
  }
  template <class M, class T>
  SWE_HD static void eval_depth(M& m, const EdgeGeom& g, const DepthState& L, const DepthState& R, double cor,
                                int cap, double* lw, double* F, const T& tape) {
    const double hl = L.h, hr = R.h;
    double ul = m.mul(L.u, g.nx) + m.mul(L.v, g.ny);
    double ur = m.mul(R.u, g.nx) + m.mul(R.v, g.ny);
    F[0] = 0.; F[1] = 0.; F[2] = 0.;
    if (!dgtc(hl + hr, kMinCapture)) return;
    double al, ar;
    W::speeds(m, ul, hl, ur, hr, &al, &ar, tape);
    // (ar - ur) hr = hr (ar - ur) and (al - ul) hl = hl (al - ul) bit for bit:
    // each product is formed once for u* and the star depth
    const double hrA = m.mul(ar - ur, hr), hlB = m.mul(al - ul, hl);
    const double hl2 = m.mul(hl, hl), hr2 = m.mul(hr, hr);
    double ustar = m.mul(hrA, ur) - m.mul(hlB, ul) + SWE_HALF(hl2 - hr2);
    ustar = SWE_DIV(ustar, hrA - hlB);
    tape.ustar(ustar);
    const double speed = plus_coriolis(cor, smax(kTol, smax(al, ar)));
    if (may_lower(g.lmin, speed, cap)) *lw = SWE_DIV(g.lmin, speed);
    // u* <= 0: the right star state, else the left one.  The side is picked
    // first and the shared formula evaluated once, so a warp whose edges take
    // both sides issues it once (the operations per side are the reference's).
    const bool right = !dgt0(ustar);
    const double hx = right ? hr : hl, ux = right ? R.u : L.u, vx = right ? R.v : L.v;
    const double ax = right ? ar : al, hxa = right ? hrA : hlB;  // hx (ax - u_n,x)
    // tangential velocity of that side
    const double vt = m.mul(ux, g.tx) + m.mul(vx, g.ty);
    double Ux[3] = {hx, m.mul(hx, ux), m.mul(hx, vx)};
    double us = m.mul(vt, g.tx) + m.mul(ustar, g.ty);
    double vs = m.mul(vt, g.nx) + m.mul(ustar, g.ny);
    double hs = SWE_DIV(hxa, ax - ustar);
    double Us[3] = {hs, m.mul(hs, us), m.mul(hs, vs)};
    double Fx[3];
    elem_flux_hh(m, g.nx, g.ny, Ux[0], Ux[1], Ux[2], right ? hr2 : hl2, Fx);
    double s = right ? smax(0., ar) : smin(0., al);
#pragma unroll
    for (int q = 0; q < 3; ++q) F[q] = Fx[q] + m.mul(s, Us[q] - Ux[q]);
  }
};

// ------------------------------------------------------- ordered doubles
// Monotone map of doubles to unsigned 64-bit keys (for non-NaN values), so
// that integer atomicMax / atomicMin give the exact floating-point max / min.
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ unsigned long long order_key(double d) {
  const unsigned long long u = (unsigned long long)dbits(d);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double order_val(unsigned long long k) {
  return dfrom((long long)((k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k));
}
#else
SWE_HD unsigned long long order_key(double d) {
  union {
    double d;
    unsigned long long u;
  } c;
  c.d = d;
  return (c.u >> 63) ? ~c.u : (c.u | 0x8000000000000000ull);
}
SWE_HD double order_val(unsigned long long k) {
  union {
    double d;
    unsigned long long u;
  } c;
  c.u = (k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
  return c.d;
}
#endif

}  // namespace swe
