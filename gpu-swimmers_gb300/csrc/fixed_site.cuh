// fixed_site.cuh -- the FP64 lattice's collision and moments in 64-bit integers.
//
// GB300 issues two FP64 operations per clock and SM, 64 integer ones.  The
// FP64 collision of a site (165 FP64 instructions and a division) took 5.16 ms
// per step at 256^3, 8 times what its bytes take, with the FP64 pipe busy 86%
// of the time; CalcHydro took 1.55 ms, 3.6 times its bytes'.  In integers they
// take 0.73 ms (0.82 of the copy bandwidth; 0.86 ms with a force, 1330
// instructions per warp, the integer pipe 73% busy) and 0.435 ms (the copy
// bandwidth).
// Here a site's 15 distributions become integers in units of 2^-59 of the
// binade of its rest population (2^-62 at density 1, 8 units to the last bit
// of a corner population), which holds every double of the site exactly unless
// it lies more than 2^7 below the rest population.  Sums are then exact, and a
// product of two 64-bit numbers takes three 32-bit multiply-adds
// (mul_hi below), good to a unit.  Mass and momentum are conserved exactly
// by the integers (the rest and the axis populations take what the divisions
// leave over); the only rounding of note is the last one, to nearest even, back
// to FP64.  Against 113-bit arithmetic the results are off by half a last
// bit, where FP64 arithmetic is off by several.
//
// Sites that do not fit (a population negative, zero, subnormal or non-finite,
// above the rest population's binade or 2^8 below it (a corner's equilibrium
// is 2^4 to 2^6 below); a velocity component of
// 1/2 or more; a force of more than about a sixteenth of the rest population) are left to FP64
// arithmetic by the callers.
#pragma once
#include "lbswim_device.cuh"

namespace lbswim {

// A 64-bit integer as two signed 32-bit digits: v = h 2^32 + l.
struct Digits {
  int h, l;
};
__host__ __device__ __forceinline__ Digits digits(long long v) {
  const unsigned l = (unsigned)(unsigned long long)v;
  unsigned h = (unsigned)((unsigned long long)v >> 32);
  // l < 0 borrows one from the high digit: h + (2 l >> 32), one multiply-add
#ifdef __CUDA_ARCH__
  asm("mad.hi.u32 %0, %1, 2, %2;" : "=r"(h) : "r"(l), "r"(h));
#else
  h += l >> 31;
#endif
  return Digits{(int)h, (int)l};
}

// a b / 2^64 rounded to nearest, but for the product of the low digits, which is
// left out (within a quarter, of either sign).  |a|, |b| < 2^63 - 2^31; the sum of the
// cross products must stay below 2^63.
__host__ __device__ __forceinline__ long long mul_hi(Digits a, Digits b) {
  const long long t = 0x80000000ll + (long long)a.h * b.l + (long long)a.l * b.h;
  return (long long)a.h * b.h + (t >> 32);
}
// The same of a b + c d.
__host__ __device__ __forceinline__ long long mul_hi2(Digits a, Digits b, Digits c, Digits d) {
  const long long t = 0x80000000ll + (long long)a.h * b.l + (long long)a.l * b.h +
                      (long long)c.h * d.l + (long long)c.l * d.h;
  return (long long)a.h * b.h + (long long)c.h * d.h + (t >> 32);
}
// x / 3, x / 9 and x / 24, |x| < 2^63 - 2^31, within a unit.
__host__ __device__ __forceinline__ long long third_of(long long x) {
  return mul_hi(digits(x), Digits{0x55555555, 0x55555555});
}
__host__ __device__ __forceinline__ long long ninth_of(long long x) {
  return mul_hi(digits(x), Digits{0x1c71c71c, 0x71c71c72});
}
__host__ __device__ __forceinline__ long long d24th_of(long long x) {
  return mul_hi(digits(x), Digits{0x0aaaaaab, (int)0xaaaaaaab});
}

__host__ __device__ __forceinline__ unsigned hi_word(unsigned long long v) {
  return (unsigned)(v >> 32);
}
__host__ __device__ __forceinline__ int leading_zeros(unsigned v) {  // v != 0
#ifdef __CUDA_ARCH__
  int n;
  asm("bfind.shiftamt.u32 %0, %1;" : "=r"(n) : "r"(v));
  return n;
#else
  return v ? __builtin_clz(v) : 32;
#endif
}
__host__ __device__ __forceinline__ unsigned long long double_bits(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned long long)__double_as_longlong(x);
#else
  unsigned long long b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
__host__ __device__ __forceinline__ double bits_double(unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}

// Units of a site: 2^(k - 1082), k the biased exponent of its rest population.
constexpr int FIXED_MAX_DROP = 7;  // lowest population's binade below the rest population's
constexpr int FIXED_MIN_K = 128, FIXED_MAX_K = 1920;  // no result leaves the normal doubles

// The 15 distributions as integers below 2^60 (exactly), k from d[0]; false
// when the site does not fit.
__host__ __device__ __forceinline__ bool site_to_fixed(const double d[15],
                                                       unsigned long long X[15], int& k) {
  const unsigned long long b0 = double_bits(d[0]);
  k = (int)(hi_word(b0) >> 20);  // with the sign: a negative d[0] gives k >= 2048
  unsigned any = 0u;
#pragma unroll
  for (int p = 0; p < 15; ++p) {
    const unsigned long long b = double_bits(d[p]);
    // MAX_DROP less the binades below the rest population's, 0 to 7 when it fits;
    // sign, zero, inf and nan wrap to a large value
    const unsigned up = (hi_word(b) >> 20) - (unsigned)(k - FIXED_MAX_DROP);
    any |= up;
    const unsigned h = (hi_word(b) & 0xfffffu) | 0x100000u, l = (unsigned)b;
#ifdef __CUDA_ARCH__
    X[p] = ((unsigned long long)__funnelshift_l(l, h, up) << 32) | __funnelshift_l(0u, l, up);
#else
    X[p] = (((unsigned long long)h << 32) | l) << (up & 31u);
#endif
  }
  static_assert((FIXED_MAX_DROP & (FIXED_MAX_DROP + 1)) == 0, "a mask tests the drops");
  return any <= (unsigned)FIXED_MAX_DROP && k >= FIXED_MIN_K && k <= FIXED_MAX_K;
}

// x in the units of k, to nearest (a force of 1e-8 has 36 bits of units at density 1, and
// a steady one cut toward zero would lose momentum at every step); false when
// |x| >= 2^56 units (a sixteenth of the top of the rest population's binade) or not
// finite.
__host__ __device__ __forceinline__ bool value_to_fixed(double x, int k, long long& v) {
  const unsigned long long b = double_bits(x);
  const int e = (int)((hi_word(b) >> 20) & 0x7ffu);
  const int drop = k - e;
  const int s = drop + 4 < 65 ? drop + 4 : 65;  // 8 .. 65 when it fits
  const unsigned long long m = (b << 11) | 0x8000000000000000ull;
  const long long a = (long long)((((m >> 1) >> ((s - 2) & 63)) + 1) >> 1);
  const long long sg = (long long)b >> 63;
  v = (a ^ sg) - sg;
  return drop >= 4;
}

// The double nearest to M 2^(1 - lz) units of k, bit 62 of M the top one set
// (ties to even).
__host__ __device__ __forceinline__ double round_to_double(unsigned long long M, int lz, int k) {
  // to a multiple of 2^10: half of one, less a bit unless that ends on an even one
  const unsigned long long r = M + (0x1ffu + (((unsigned)M >> 10) & 1u));
  // bit 63 of the units is the binade k + 4; bit 52 of r >> 10 carries into
  // the exponent field, and so does a mantissa rounded up to 2^53
  const unsigned long long m = r >> 10;
  const unsigned h = hi_word(m) + ((unsigned)(k + 3) << 20) - ((unsigned)lz << 20);
  return bits_double(((unsigned long long)h << 32) | (unsigned)m);
}
// The double nearest to X units of k, 2^32 <= X < 2^63.
__host__ __device__ __forceinline__ double fixed_to_double(unsigned long long X, int k) {
  const int lz = leading_zeros(hi_word(X));
  return round_to_double(X << ((lz - 1) & 31), lz, k);
}
// The same for any |X| < 2^63.
__host__ __device__ __forceinline__ double signed_fixed_to_double(long long X, int k) {
  if (X == 0) return 0.0;
  const unsigned long long sg = (unsigned long long)(X >> 63);
  const unsigned long long a = ((unsigned long long)X ^ sg) - sg;
  const unsigned h = hi_word(a);
  const int lz = h ? leading_zeros(h) : 32 + leading_zeros((unsigned)a);
  const double r = round_to_double(a << ((lz - 1) & 63), lz, k);
  return bits_double(double_bits(r) | (sg & 0x8000000000000000ull));
}

// 1 / r in units of 2^-61, r = R 2^lz / 2^64 in [1/2, 1) with lz the leading
// zeros of R >= 2^59, relative error below 2^-59: a 23-bit reciprocal,
// then two Newton steps x + x (1 - r x).
__host__ __device__ __forceinline__ long long fixed_reciprocal(unsigned long long R, int& lz) {
  lz = leading_zeros(hi_word(R));
  const unsigned long long Rn = R << (lz & 31);
  const unsigned rh = hi_word(Rn), rl = (unsigned)Rn;
  const float rf = (float)(rh >> 8) * 0x1p-24f;  // exact
#ifdef __CUDA_ARCH__
  float xf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(xf) : "f"(rf));
#else
  const float xf = 1.0f / rf;
#endif
  // x in units of 2^-30; r = 1/2 would give 2^31
  unsigned x0 = (unsigned)(xf * 0x1p30f);
  x0 = x0 < 0x7fffffffu ? x0 : 0x7fffffffu;
  // 1 - r x in units of 2^-62 (below 2^42), then of 2^-61 (below 2^21)
  const long long e0 = (1ll << 62) -
                       (long long)((unsigned long long)rh * x0 +
                                   (((unsigned long long)rl * x0) >> 32));
  const long long x1 =
      (long long)((unsigned long long)x0 << 31) + (((long long)(int)x0 * (int)(e0 >> 12)) >> 19);
  const unsigned h1 = hi_word((unsigned long long)x1), l1 = (unsigned)x1;
  const long long e1 = (1ll << 61) -
                       (long long)((unsigned long long)rh * h1 +
                                   (((unsigned long long)rh * l1) >> 32) +
                                   (((unsigned long long)rl * h1) >> 32));
  return x1 + (((long long)(int)h1 * (int)e1) >> 29);
}

// The relaxation constants of a lattice for site_collide_fixed.
struct FixedRelax {
  Digits ws;     // omega_s - 1 in units of 2^-63
  Digits wb;     // omega_b - 1
  Digits fs;     // force_s / 2
  Digits fb;     // (force_b / force_s - 4) / 8
  int usable;    // 0: a constant does not fit (relaxation times not above 0 or
                 // beyond 2^28, or their forcing factors more than 8 apart)
};

// v in units of 2^-63; false when |v| leaves no room for the digits' carry.
inline bool fixed_const(double v, Digits& d) {
  const bool fits = v >= -0x1.fffffffp-1 && v <= 0x1.fffffffp-1;
  if (fits) d = digits((long long)(v * 0x1p63));
  return fits;
}
inline FixedRelax make_fixed_relax(const Relax<double>& k) {
  FixedRelax c{};
  // (force_b / force_s - 4) / 8 is at most 1/2 in the kernel's bounds
  const double ratio = k.force_s > 0.0 ? k.force_b / k.force_s : -1.0;
  c.usable = ratio >= 0.0 && ratio <= 8.0 && fixed_const(k.omega_s - 1.0, c.ws) &&
             fixed_const(k.omega_b - 1.0, c.wb) && fixed_const(0.5 * k.force_s, c.fs) &&
             fixed_const((ratio - 4.0) * 0.125, c.fb);
  return c;
}

// Density and momentum of the integers (R < 15 2^60, unsigned).
__host__ __device__ __forceinline__ void hydro_fixed(const unsigned long long X[15],
                                                     unsigned long long& R, long long& jx,
                                                     long long& jy, long long& jz) {
  const unsigned long long c1 = X[7] + X[8], c2 = X[9] + X[10], c3 = X[11] + X[12],
                           c4 = X[13] + X[14];
  const unsigned long long xp = c1 + c2, xm = c3 + c4;
  R = X[0] + (X[1] + X[2]) + (X[3] + X[4]) + (X[5] + X[6]) + (xp + xm);
  jx = (long long)((X[1] - X[2]) + (xp - xm));
  jy = (long long)((X[3] - X[4]) + ((c1 - c2) + (c3 - c4)));
  jz = (long long)((X[5] - X[6]) +
                   (((X[7] - X[8]) + (X[9] - X[10])) + ((X[11] - X[12]) + (X[13] - X[14]))));
}

// The collision of lb.cu:121-203 (collide() in lbswim_device.cuh) on integers:
// X in, post-collision X out.  FORCED: F holds the force in the same units.
// With w' = omega - 1, q_ab = rho u_a u_b, q = rho u.u, F' = force_s F and
// t the traceless stress the relaxed moments are
//   off the diagonal  S'_ab = q_ab + w'_s (q_ab - S_ab) + u_a F'_b + F'_a u_b
//   traceless         T_a = P_a + w'_s (P_a - t_a) + 2 (u_a F'_a - u.F'/3), P_a = q_aa - q/3
//   trace             Tr = -q + w'_b (q - TrS) - 2 w'_s q + (force_b/force_s - 4) u.F'
// and the populations R/72 + Tr/24 +- J/24 +- S'/8 (corners), R/9 + T_a/2 +- J_a/3
// (axes), and the rest.  False when a velocity or a result does not fit.
template <bool FORCED>
__host__ __device__ __forceinline__ bool site_collide_fixed(unsigned long long X[15],
                                                            const long long F[3],
                                                            const FixedRelax& c) {
  typedef unsigned long long U;
  // moments
  const U a = X[1] + X[2], b = X[3] + X[4], cc = X[5] + X[6];
  const U P1 = X[7] + X[8], M1 = X[7] - X[8], P2 = X[9] + X[10], M2 = X[9] - X[10];
  const U P3 = X[11] + X[12], M3 = X[11] - X[12], P4 = X[13] + X[14], M4 = X[13] - X[14];
  const U PPp = P1 + P2, PMp = P1 - P2, MPp = M1 + M2, MMp = M1 - M2;
  const U PPm = P3 + P4, PMm = P3 - P4, MPm = M3 + M4, MMm = M3 - M4;
  const U sum = PPp + PPm, A3 = a + b + cc;
  const U R = X[0] + A3 + sum;
  const long long jx = (long long)((X[1] - X[2]) + (PPp - PPm));
  const long long jy = (long long)((X[3] - X[4]) + (PMp + PMm));
  const long long jz = (long long)((X[5] - X[6]) + (MPp + MPm));
  const long long Sxy = (long long)(PMp - PMm), Sxz = (long long)(MPp - MPm),
                  Syz = (long long)(MMp + MMm);
  // A corner sum (R/9 near equilibrium) and rho u.u below 2^60, |u_a| < 1/2 and
  // |F_a| < 2^56 keep every intermediate, R < 2^63 among them, within 64 bits.
  unsigned worst = hi_word(sum);
  const long long th = third_of((long long)A3);
  const long long tx = (long long)a - th, ty = (long long)b - th, tz = (long long)cc - th;
  const long long TrS = (long long)(2 * sum - X[0]);
  // velocity in units of 2^-64, |u| < 1/2: |m| < R / 2 by the high words
  long long mx = jx, my = jy, mz = jz;
  if (FORCED) {
    mx += F[0] >> 1;
    my += F[1] >> 1;
    mz += F[2] >> 1;
  }
  const unsigned Rh = hi_word(R), half = Rh >> 1;
  const unsigned cx = (unsigned)(mx >> 32) + half, cy = (unsigned)(my >> 32) + half,
                 cz = (unsigned)(mz >> 32) + half;
  // 1 <= half + m_hi <= 2 half - 2 keeps |m| < R / 2
  unsigned fast = cx - 1u;
  fast = cy - 1u > fast ? cy - 1u : fast;
  fast = cz - 1u > fast ? cz - 1u : fast;
  int lz;
  const Digits y = digits(fixed_reciprocal(R, lz));
  const Digits mdx = digits(mx), mdy = digits(my), mdz = digits(mz);
  const Digits ux = digits((long long)((U)mul_hi(mdx, y) << (lz + 3)));
  const Digits uy = digits((long long)((U)mul_hi(mdy, y) << (lz + 3)));
  const Digits uz = digits((long long)((U)mul_hi(mdz, y) << (lz + 3)));
  const long long qxx = mul_hi(mdx, ux), qyy = mul_hi(mdy, uy), qzz = mul_hi(mdz, uz);
  const long long qxy = mul_hi(mdx, uy), qxz = mul_hi(mdx, uz), qyz = mul_hi(mdy, uz);
  const long long q = qxx + qyy + qzz, q3 = third_of(q);
  // a slow site's q is 0 or, rounded, just below it
  const unsigned qh = hi_word((unsigned long long)q + 64u);
  worst = qh > worst ? qh : worst;
  // relaxed stress
  long long Tx = qxx - q3, Ty = qyy - q3, Tz = qzz - q3;
  Tx += 2 * mul_hi(digits(Tx - tx), c.ws);
  Ty += 2 * mul_hi(digits(Ty - ty), c.ws);
  Tz += 2 * mul_hi(digits(Tz - tz), c.ws);
  long long nxy = qxy + 2 * mul_hi(digits(qxy - Sxy), c.ws);
  long long nxz = qxz + 2 * mul_hi(digits(qxz - Sxz), c.ws);
  long long nyz = qyz + 2 * mul_hi(digits(qyz - Syz), c.ws);
  long long Tr = 2 * mul_hi(digits(q - TrS), c.wb) - q - 4 * mul_hi(digits(q), c.ws);
  long long Jx = jx, Jy = jy, Jz = jz;
  if (FORCED) {
    const Digits fx = digits(4 * mul_hi(digits(F[0]), c.fs));
    const Digits fy = digits(4 * mul_hi(digits(F[1]), c.fs));
    const Digits fz = digits(4 * mul_hi(digits(F[2]), c.fs));
    const long long gx = mul_hi(ux, fx), gy = mul_hi(uy, fy), gz = mul_hi(uz, fz);
    const long long g = gx + gy + gz, g3 = third_of(g);
    Tx += 2 * (gx - g3);
    Ty += 2 * (gy - g3);
    Tz += 2 * (gz - g3);
    nxy += mul_hi2(ux, fy, uy, fx);
    nxz += mul_hi2(ux, fz, uz, fx);
    nyz += mul_hi2(uy, fz, uz, fy);
    Tr += 16 * mul_hi(digits(g), c.fb);
    Jx += F[0];
    Jy += F[1];
    Jz += F[2];
  }
  // populations: the corners first, then the axes with the rest of the
  // momentum, then the rest population with the rest of the mass
  const U R9 = (U)ninth_of((long long)R);
  const long long J24x = d24th_of(Jx), J24y = d24th_of(Jy), J24z = d24th_of(Jz);
  const U A = ((R9 + 4) >> 3) + (U)d24th_of(Tr);
  const U Cxy = (U)((nxy + 4) >> 3), Cxz = (U)((nxz + 4) >> 3), Cyz = (U)((nyz + 4) >> 3);
  {
    const U G = A + (U)J24x, Hy = (U)J24y + Cxy, Hz = (U)J24z + Cxz;
    const U K1 = G + Hy, K2 = G - Hy, L1 = Hz + Cyz, L2 = Hz - Cyz;
    X[7] = K1 + L1;
    X[8] = K1 - L1;
    X[9] = K2 + L2;
    X[10] = K2 - L2;
  }
  {
    const U G = A - (U)J24x, Hy = (U)J24y - Cxy, Hz = (U)J24z - Cxz;
    const U K1 = G + Hy, K2 = G - Hy, L1 = Hz + Cyz, L2 = Hz - Cyz;
    X[11] = K1 + L1;
    X[12] = K1 - L1;
    X[13] = K2 + L2;
    X[14] = K2 - L2;
  }
  // the axis pairs differ by what the corners leave of the momentum
  const U Dx = (U)Jx - 8 * (U)J24x, Dy = (U)Jy - 8 * (U)J24y, Dz = (U)Jz - 8 * (U)J24z;
  X[1] = (U)((long long)(2 * R9 + (U)Tx + Dx) >> 1);
  X[2] = X[1] - Dx;
  X[3] = (U)((long long)(2 * R9 + (U)Ty + Dy) >> 1);
  X[4] = X[3] - Dy;
  X[5] = (U)((long long)(2 * R9 + (U)Tz + Dz) >> 1);
  X[6] = X[5] - Dz;
  X[0] = R - 8 * A - (X[1] + X[2]) - (X[3] + X[4]) - (X[5] + X[6]);
  // every result in [2^32, 2^63)
  int least = 1;
#pragma unroll
  for (int p = 0; p < 15; ++p) {
    const int h = (int)hi_word(X[p]);
    least = h < least ? h : least;
  }
  return worst < (1u << 28) && fast < 2u * half - 2u && least == 1;
}

}  // namespace lbswim
