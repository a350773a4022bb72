// Integrator of the filament step and the device helpers it shares with the
// rest of the pipeline, as a header compiled by two units:
//   sc_kernels.cu      (--fmad=false): FAST = false, the reference's exact
//                      arithmetic, bit-identical to it;
//   sc_kernels_fast.cu (--fmad=true):  FAST = true, the same algorithm with
//                      contraction, one reciprocal per shared denominator and
//                      rsqrt normalisation (mixed precision only).
#pragma once

#include "sc_common.cuh"
#include "sc_pair.cuh"

namespace sc {

// ---------------------------------------------------------------------------
// Bond geometry from two sites: Bond::ReInit (src/bond.cpp:22-37) followed by
// Object::UpdatePeriodic / periodic_boundary_conditions
// (src/object.cpp:202-210, src/linear_algebra.cpp:100-117).
template <int ND>
__device__ __forceinline__ void bond_from_sites(const double *hinv,
                                                const double *r1,
                                                const double *r2, double s[3],
                                                double u[3], double &len) {
  double pos[3] = {0, 0, 0};
  u[0] = u[1] = u[2] = 0.0;
  s[0] = s[1] = s[2] = 0.0;
  len = 0;
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    u[i] = r2[i] - r1[i];
    len += u[i] * u[i];
  }
  len = sqrt(len);
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    pos[i] = r1[i] + 0.5 * u[i];
    u[i] /= len;
  }
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    s[i] = 0.0;
#pragma unroll
    for (int j = 0; j < ND; ++j) s[i] += hinv[ND * i + j] * pos[j];
    s[i] -= nint(s[i]);
  }
}

__device__ __forceinline__ int32_t to_fixed(double s) {
  // s in [-1/2, 1/2]: round(s * 2^32) wraps into int32 (1/2 and -1/2 map to
  // the same point of the periodic box).
  long long q = __double2ll_rn(s * 4294967296.0);
  return (int32_t)(uint32_t)(unsigned long long)q;
}

template <int ND>
__device__ __forceinline__ void store_geom(const DevState &d, int buf, int b,
                                           const double s[3],
                                           const double u[3], double len,
                                           int prec) {
  if (prec == 0) {
    BondGeomF64 g;
    g.s[0] = s[0];
    g.s[1] = s[1];
    g.s[2] = s[2];
    g.u[0] = u[0];
    g.u[1] = u[1];
    g.u[2] = u[2];
    g.len = len;
    g.pad = 0.0;
    d.g64[buf][b] = g;
  } else {
    BondGeomF32 g;
    g.q[0] = to_fixed(s[0]);
    g.q[1] = to_fixed(s[1]);
    g.q[2] = ND == 3 ? to_fixed(s[2]) : 0;
    g.hl = (float)(0.5 * len);
    g.u[0] = (float)u[0];
    g.u[1] = (float)u[1];
    g.u[2] = (float)u[2];
    g.pad = 0.f;
    d.g32[buf][b] = g;
  }
}

// IEEE division (round to nearest) by a shared reciprocal, for the exact
// integrator: several quotients have one divisor, and a quotient's chain is
// the integrator's critical path.  y = RN(1/b) from the hardware's approximate
// reciprocal by one third-order step, which leaves it within one ulp, and
// Markstein's correction y + y (1 - b y), whose result is the correctly
// rounded reciprocal unless b's significand is all ones (Markstein, IBM J.
// Res. Dev. 34:111-119, 1990; Muller et al., Handbook of Floating-Point
// Arithmetic, 2nd ed., sec. 4.7).  A quotient starts as q0 = x y, within two
// ulps of x/b; one correction q1 = q0 + y (x - b q0) makes it faithful, and a
// second one on a faithful quotient is correctly rounded (the same theorem:
// x - b q1 is exact); a zero x keeps q0, a zero of the quotient's sign.  The
// result has the bits of x / b where `ok` holds at the end: every exponent
// leaves room for the intermediates, and no divisor's significand is all ones.
// The caller repeats its work with the compiler's division where it does not,
// so that no quotient pays for a branch.  Measured, one warp: 126 cycles for
// the compiler's division (two independent ones do not overlap: 262); here 61
// for y and 47 for each quotient, which do.
__device__ __forceinline__ bool mid_exponent(double x) {
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  return e - (1023u - 450u) < 900u;
}
__device__ __forceinline__ double recip_rn(double b, bool &ok) {
  const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
  ok = ok && mid_exponent(b) && !(lo == 0xffffffffu && (hi & 0xfffffu) == 0xfffffu);
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  double e = __fma_rn(-b, y, 1.0);
  y = __fma_rn(y, __fma_rn(e, e, e), y);
  e = __fma_rn(-b, y, 1.0);
  return __fma_rn(e, y, y);
}
__device__ __forceinline__ double div_rn(double x, double b, double y, bool &ok) {
  const bool zero = x == 0.0;
  ok = ok && (mid_exponent(x) || zero);
  const double q0 = __dmul_rn(x, y);
  const double q1 = __fma_rn(__fma_rn(-b, q0, x), y, q0);
  const double q2 = __fma_rn(__fma_rn(-b, q1, x), y, q1);
  return zero ? q0 : q2;
}
// One quotient by a divisor whose RN(1/b) is at hand.
__device__ __forceinline__ double div_by(double x, double b, double y) {
  bool ok = mid_exponent(b);
  const double q = div_rn(x, b, y, ok);
  if (ok) return q;
  asm volatile("" : "+d"(x));  // a branch: not computed beside the fast path
  return x / b;
}

__device__ __forceinline__ void cross3(const double *a, const double *b,
                                       double *c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}

__device__ __forceinline__ void kahan_add(float &sum, float &comp, float x) {
  float y = x - comp;
  float t = sum + y;
  comp = (t - sum) - y;
  sum = t;
}

// Sum of one bond's crosslink anchor contributions in link order, as
// CrosslinkSpecies::ApplyCrosslinkTetherForces adds them to Bond::force_ /
// torque_ before the pair path (src/crosslink_species.cpp:260-266,
// src/anchor.cpp:132-146): ND force components, 3 torque components.  Of
// the anchors listed on the bond, those that sit on it count.
template <int ND>
__device__ __forceinline__ void bond_xlink_sum(const DevState &d, int b, double F[3],
                                               double T[3]) {
  const int e0 = d.xb_off[b], e1 = d.xb_off[b + 1];
  for (int e = e0; e < e1; ++e) {
    const double2 *c = reinterpret_cast<const double2 *>(d.xl_c) + 4 * (size_t)d.xb_ent[e];
    if ((int)c[3].x != b) continue;
    const double2 v0 = c[0], v1 = c[1], v2 = c[2];
    F[0] += v0.x;
    F[1] += v0.y;
    if (ND == 3) F[2] += v1.x;
    T[0] += v1.y;
    T[1] += v2.x;
    T[2] += v2.y;
  }
}

// Bond::force_ / torque_ after Interact: crosslink anchors first, then the
// bond's pair contributions in slot (= pair) order.  FP64 sums as the
// reference accumulates them; in mixed precision FP32 sums with Kahan
// compensation, added to the FP64 crosslink sum.  A pair slot is 8 values: force (3), torque (3),
// padding (2).  [e0, e1) is the bond's slot range (e_off, e_off + e_cnt),
// which the integrators load before they wait for the pair stage: the
// rebuild wrote it, before the pair stage ran.
template <int ND, int PREC>
__device__ __forceinline__ void bond_pair_sum(const DevState &d, int b, int e0, int e1,
                                              double F[3], double T[3]) {
  F[0] = F[1] = F[2] = 0.0;
  T[0] = T[1] = T[2] = 0.0;
  if (d.nx) bond_xlink_sum<ND>(d, b, F, T);
  // Slots are loaded in batches whose loads are all in flight together, then
  // added in order: bound by the round trips to L2, one after another in a
  // plain loop's remainder, and most bonds have one to five slots.  20,000
  // filaments of 5 to 200 bonds, 20 mixed steps: 9.45 ms before, 8.97 ms now.
  if (PREC == 0) {
    constexpr int BATCH = 3;
    const double2 *c = reinterpret_cast<const double2 *>(d.cf64) + 4 * (size_t)e0;
    for (int e = e0; e < e1; e += BATCH, c += 4 * BATCH) {
      double2 v[BATCH][3];
#pragma unroll
      for (int q = 0; q < BATCH; ++q)
        if (e + q < e1) {
          v[q][0] = c[4 * q];
          v[q][1] = c[4 * q + 1];
          v[q][2] = c[4 * q + 2];
        }
#pragma unroll
      for (int q = 0; q < BATCH; ++q)
        if (e + q < e1) {
          F[0] += v[q][0].x;
          F[1] += v[q][0].y;
          if (ND == 3) F[2] += v[q][1].x;
          T[0] += v[q][1].y;
          T[1] += v[q][2].x;
          T[2] += v[q][2].y;
        }
    }
  } else {
    constexpr int BATCH = 4;
    float sF[3] = {0.f, 0.f, 0.f}, cF[3] = {0.f, 0.f, 0.f};
    float sT[3] = {0.f, 0.f, 0.f}, cT[3] = {0.f, 0.f, 0.f};
    const float4 *c = reinterpret_cast<const float4 *>(d.cf32) + 2 * (size_t)e0;
    for (int e = e0; e < e1; e += BATCH, c += 2 * BATCH) {
      float4 v[BATCH][2];
#pragma unroll
      for (int q = 0; q < BATCH; ++q)
        if (e + q < e1) {
          v[q][0] = c[2 * q];
          v[q][1] = c[2 * q + 1];
        }
#pragma unroll
      for (int q = 0; q < BATCH; ++q)
        if (e + q < e1) {
          kahan_add(sF[0], cF[0], v[q][0].x);
          kahan_add(sF[1], cF[1], v[q][0].y);
          if (ND == 3) kahan_add(sF[2], cF[2], v[q][0].z);
          kahan_add(sT[0], cT[0], v[q][0].w);
          kahan_add(sT[1], cT[1], v[q][1].x);
          kahan_add(sT[2], cT[2], v[q][1].y);
        }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      F[i] += (double)sF[i] - (double)cF[i];
      T[i] += (double)sT[i] - (double)cT[i];
    }
  }
}

// Bond::force_ / torque_ of the mixed step with the pair stage fused in.
// The bond evaluates each of its pairs itself (pair_force_f32 on both bonds'
// FP32 geometry of this step), in entry (= slot) order, and adds its side of
// the force and torque exactly as bond_pair_sum adds the slots the pair stage
// would have written: the same values in the same order, so the same bits.
// Both bonds of a pair evaluate it.  The first (role 0) stores the force, and
// only when it was computed; the second reads the stored force only when it
// was not, so no bond reads a value that another is writing for this step.
template <int ND>
__device__ __forceinline__ void bond_pair_eval_sum(const SysConst &k, const DevState &d,
                                                   const float *hf, int rbuf, int b,
                                                   double F[3], double T[3]) {
  const int e0 = d.e_off[b], e1 = e0 + d.e_cnt[b];
  F[0] = F[1] = F[2] = 0.0;
  T[0] = T[1] = T[2] = 0.0;
  if (d.nx) bond_xlink_sum<ND>(d, b, F, T);
  float sF[3] = {0.f, 0.f, 0.f}, cF[3] = {0.f, 0.f, 0.f};
  float sT[3] = {0.f, 0.f, 0.f}, cT[3] = {0.f, 0.f, 0.f};
  for (int e = e0; e < e1; ++e) {
    const int ent = d.e_ent[e], p = ent >> 1;
    const BondGeomF32 A = d.g32[rbuf][d.pa[p]], B = d.g32[rbuf][d.pb[p]];
    float4 *stale = reinterpret_cast<float4 *>(d.pf32) + (size_t)p;
    float f[3], t1[3], t2[3], v[6];
    const bool set = pair_force_f32<ND>(k, hf, A, B, *stale, f, t1, t2);
    if (ent & 1) {
      v[0] = -f[0];
      v[1] = -f[1];
      v[2] = -f[2];
      v[3] = -t2[0];
      v[4] = -t2[1];
      v[5] = -t2[2];
    } else {
      if (set) *stale = make_float4(f[0], f[1], f[2], 0.f);
      v[0] = f[0];
      v[1] = f[1];
      v[2] = f[2];
      v[3] = t1[0];
      v[4] = t1[1];
      v[5] = t1[2];
    }
    kahan_add(sF[0], cF[0], v[0]);
    kahan_add(sF[1], cF[1], v[1]);
    if (ND == 3) kahan_add(sF[2], cF[2], v[2]);
    kahan_add(sT[0], cT[0], v[3]);
    kahan_add(sT[1], cT[1], v[4]);
    kahan_add(sT[2], cT[2], v[5]);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    F[i] += (double)sF[i] - (double)cF[i];
    T[i] += (double)sT[i] - (double)cT[i];
  }
}

// ---------------------------------------------------------------------------
// Integrator.  A block holds a run of whole filaments, one thread per site,
// filaments back to back.  Per-site work runs in parallel; the sequential
// recurrences of one filament (metric determinants, Thomas solves,
// renormalisation) run on one dedicated lane per filament (lane lf for
// filament lf of the block, lane C/2 + lf for the backward determinant), so
// a block's serial work occupies one or two warps instead of every warp.

// The reference's tridiagonal_solver (Thomas, src/linear_algebra.cpp:164-197)
// in two parts, its operations in its order, so its bits: the elimination of
// the matrix (den_i = b_i - a_{i-1} c'_{i-1}, c'_i = c_i / den_i) and the
// elimination and back substitution of a right-hand side (d'_i = (d_i -
// a_{i-1} d'_{i-1}) / den_i).  Split, the matrix part of every system and the
// determinants run at once on different lanes, before the forces are known,
// and a right-hand side's chain holds a quotient by a known reciprocal instead
// of a division.  Bound by that serial chain: inside the integrator of 21-site
// filaments 250 cycles a row for the matrices with the determinants and 145 a
// right-hand side, where one solve with the compiler's division took 346 and
// the determinants 85.  Operands are loaded a row ahead of the chain.  The
// matrices are symmetric with couplings h (h_i couples rows i and i + 1; NEG:
// -h_i); DIAG2: every diagonal element is 2.
template <bool NEG, bool DIAG2>
__device__ __forceinline__ void tridiag_factor_ieee(const double *h, const double *b, double *den,
                                                    double *inv, double *up, int m) {
  double cp = 0.0;
  for (int i = 0; i < m; ++i) {
    const double bi = DIAG2 ? 2.0 : b[i];
    const double a = i > 0 ? (NEG ? -h[i - 1] : h[i - 1]) : 0.0;
    const double dd = i > 0 ? bi - a * cp : bi;
    den[i] = dd;
    inv[i] = 1.0 / dd;
    if (i < m - 1) up[i] = cp = (NEG ? -h[i] : h[i]) / dd;
  }
}
// A shared-memory array named by its 32-bit address, for the routines below:
// they are functions of their own, so that their loops keep their registers
// (inlined into the integrators, at their register caps, a row took twice as
// long), and take addresses that are known to be shared memory's.
typedef unsigned sptr;
__device__ __forceinline__ sptr to_sptr(const double *p) {
  return (sptr)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ double *of_sptr(sptr a) {
  return static_cast<double *>(__cvta_shared_to_generic(a));
}

template <bool NEG>
static __device__ __noinline__ void tridiag_rhs_fn(sptr ah, sptr aden, sptr ainv, sptr aup, sptr ad,
                                            sptr ax, int m) {
  const double *h = of_sptr(ah), *den = of_sptr(aden), *inv = of_sptr(ainv), *up = of_sptr(aup);
  const double *d = of_sptr(ad);
  double *x = of_sptr(ax);
  bool ok = true;
  double v = div_rn(d[0], den[0], inv[0], ok);
  x[0] = v;
  double hn = h[0], dn = d[1], bn = den[1], yn = inv[1];
  for (int i = 1; i < m; ++i) {
    const double a = NEG ? -hn : hn, di = dn, bi = bn, yi = yn;
    if (i + 1 < m) {
      hn = h[i];
      dn = d[i + 1];
      bn = den[i + 1];
      yn = inv[i + 1];
    }
    v = div_rn(di - a * v, bi, yi, ok);
    x[i] = v;
  }
  if (!ok) {
    v = d[0] / den[0];
    x[0] = v;
    for (int i = 1; i < m; ++i) {
      const double a = NEG ? -h[i - 1] : h[i - 1];
      v = (d[i] - a * v) / den[i];
      x[i] = v;
    }
  }
  double cn = up[m - 2];
  dn = x[m - 2];
  for (int i = m - 2; i >= 0; --i) {
    const double ci = cn, di = dn;
    if (i > 0) {
      cn = up[i - 1];
      dn = x[i - 1];
    }
    v = di - ci * v;
    x[i] = v;
  }
}

template <bool NEG>
__device__ __forceinline__ void tridiag_rhs(const double *h, const double *den, const double *inv,
                                            const double *up, const double *d, double *x, int m) {
  tridiag_rhs_fn<NEG>(to_sptr(h), to_sptr(den), to_sptr(inv), to_sptr(up), to_sptr(d), to_sptr(x),
                      m);
}

// Two recurrences of one filament of n sites side by side on one lane, for
// the exact step: the elimination of a matrix (mat: none without it) and a
// metric determinant of CalculateBendingForces (src/filament.cpp:627-660) --
// TRAIL: det_b from the head, to dt[n] .. dt[1]; else det_t from the tail, to
// dt[0] .. dt[n - 1].  The projection matrix (2, -cos) goes with det_t, the
// tension matrix with det_b, so lanes of both kinds run one instruction stream.
static __device__ __noinline__ void factor_and_minors_fn(bool trail, bool mat, sptr acz, sptr aoff,
                                                  sptr adiag, sptr aden, sptr ainv, sptr aup,
                                                  sptr adt, int n) {
  const double *cz = of_sptr(acz), *off = of_sptr(aoff), *diag = of_sptr(adiag);
  double *den = of_sptr(aden), *inv = of_sptr(ainv), *up = of_sptr(aup), *dt = of_sptr(adt);
  const int m = n - 1;  // rows
  const double *h = trail ? off : cz;
  const double sg = mat ? (trail ? 1.0 : -1.0) : 0.0;
  double x0 = 1.0, x1 = 2.0;
  dt[trail ? n : 0] = x0;
  dt[trail ? n - 1 : 1] = x1;
  double c = cz[trail ? n - 3 : 0];
  double hi = sg * h[0], hn = m > 2 ? sg * h[1] : 0.0;
  double bn = trail ? diag[1] : 2.0;
  bool ok = true;
  double dd = trail ? diag[0] : 2.0;
  double y = recip_rn(dd, ok);
  double cp = div_rn(hi, dd, y, ok);
  if (mat) {
    den[0] = dd;
    inv[0] = y;
    up[0] = cp;
  }
  for (int i = 1; i < m; ++i) {  // row i, minor i + 1
    const double ai = hi, bi = bn, ci = hn;
    hi = hn;
    if (i + 1 < m) bn = trail ? diag[i + 1] : 2.0;
    hn = i + 2 < m ? sg * h[i + 1] : 0.0;
    const double cn = i + 2 < n ? cz[trail ? n - i - 3 : i] : 0.0;
    const double x2 = 2 * x1 - c * c * x0;
    dt[trail ? n - i - 1 : i + 1] = x2;
    x0 = x1;
    x1 = x2;
    c = cn;
    dd = bi - ai * cp;
    y = recip_rn(dd, ok);
    cp = div_rn(ci, dd, y, ok);
    if (mat) {
      den[i] = dd;
      inv[i] = y;
      up[i] = cp;
    }
  }
  if (mat && !ok) {
    if (trail) tridiag_factor_ieee<false, false>(off, diag, den, inv, up, m);
    else tridiag_factor_ieee<true, true>(cz, nullptr, den, inv, up, m);
  }
}
__device__ __forceinline__ void factor_and_minors(bool trail, bool mat, const double *cz,
                                                  const double *off, const double *diag,
                                                  double *den, double *inv, double *up,
                                                  double *dt, int n) {
  factor_and_minors_fn(trail, mat, to_sptr(cz), to_sptr(off), to_sptr(diag), to_sptr(den),
                       to_sptr(inv), to_sptr(up), to_sptr(dt), n);
}

// 1/x for the fast integrator: from the hardware's FP64 approximate
// reciprocal y of x (PTX rcp.approx.ftz.f64), one step of the third-order
// iteration y <- y (1 + e + e^2) with e = 1 - x y, the truncated series of
// y / (1 - e) (Muller et al., Handbook of Floating-Point Arithmetic, 2nd
// ed., sec. 4.7).  The seed's relative error is below 2^-19 (measured
// 9.9e-7), so the step leaves e^3 < 2^-57 before the final rounding: within
// an ulp of 1/x, from three dependent FMAs after one approximation and no
// FP32 round trip (conversions are slow on this part).  For normal |x|,
// which the diagonals, determinants and lengths it serves are.
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ double recip_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// x^-1/2 for the fast integrator, the same way: the hardware's approximate
// inverse square root y (PTX rsqrt.approx.ftz.f64), e = 1 - x y^2, and
// y (1 - e)^-1/2 by its series to the second order, y (1 + e/2 + 3e^2/8):
// relative error about 5e^3/16 before the final rounding (seed error below
// 2^-19, measured 9.2e-7; the result within an ulp of 1/sqrt(x)).
__device__ __forceinline__ double rsqrt_nr(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y * y, 1.0);
  return fma(y, e * fma(e, 0.375, 0.5), y);
}

// ((double)w + 0.5) * 2^-32 - 0.5 for a 32-bit Philox word w, the noise's
// uniform on (-1/2, 1/2).  w + 1/2 is formed exactly from bits -- 2^51 + w +
// 1/2 is the double with exponent 51 and mantissa 2w + 1 -- instead of by an
// integer-to-double conversion; the product with 2^-32 is exact, so the
// result has the same bits as the expression above.
__device__ __forceinline__ double centered_uniform(uint32_t w) {
  const double h =
      __longlong_as_double(0x4320000000000000ll | (((long long)w << 1) | 1ll)) - 2251799813685248.0;
  return h * 2.3283064365386963e-10 - 0.5;
}

// The same uniform in FP32 from the word's top 23 bits, (m + 1/2) 2^-23 -
// 1/2 with m = w >> 9, exact (m from its bits, as above): the mixed step's
// noise, within 2^-24 of the FP64 one.
__device__ __forceinline__ float centered_uniform_f(uint32_t w) {
  const float m = __uint_as_float(0x4B000000u | (w >> 9)) - 8388608.0f;
  return fmaf(m + 0.5f, 1.1920928955078125e-7f, -0.5f);
}

__device__ __forceinline__ double recip_t(double x) { return recip_nr(x); }
__device__ __forceinline__ float recip_t(float x) { return rcp_approx(x); }

// FAST: one reciprocal per row instead of two divisions (FP64: recip_nr;
// FP32: the approximate reciprocal, within an ulp).  Each row's operands are
// loaded a row ahead of the chain.
template <class T>
__device__ __forceinline__ void thomas_fast(T *a, const T *b, T *c, T *d, int n) {
  n--;
  T r = recip_t(b[0]);
  T cp = c[0] * r;
  T dp = d[0] * r;
  T an = a[0], bn = b[1], cn = n > 1 ? c[1] : T(0), dn = d[1];
  c[0] = cp;
  d[0] = dp;
  for (int i = 1; i < n; ++i) {
    const T am = an, bi = bn, ci = cn, di = dn;
    an = a[i];
    bn = b[i + 1];
    cn = i + 1 < n ? c[i + 1] : T(0);
    dn = d[i + 1];
    r = recip_t(bi - am * cp);
    cp = ci * r;
    dp = (di - am * dp) * r;
    c[i] = cp;
    d[i] = dp;
  }
  dp = (dn - an * dp) * recip_t(bn - an * cp);
  d[n] = dp;
  cn = c[n - 1];
  dn = d[n - 1];
  for (int i = n - 1; i >= 0; --i) {
    const T ci = cn, di = dn;
    if (i > 0) {
      cn = c[i - 1];
      dn = d[i - 1];
    }
    dp = di - ci * dp;
    d[i] = dp;
  }
}

// Two-sided ("twisted") elimination of one tridiagonal system of n rows for
// the fast integrator (van der Vorst, "Large tridiagonal and block
// tridiagonal linear systems on vector and parallel computers", Parallel
// Computing 5:45-54, 1987): a pair of lanes of one warp, the top lane
// eliminating rows 0..m-1 downwards and the bottom lane rows n-1..m+1
// upwards, meet at row m = n/2, then substitute back outwards.  Half the
// sequential depth of thomas_fast, the same layout (row r: lower coefficient
// a[r-1], diagonal b[r], upper c[r], right-hand side d[r]); the solution
// ends in d.  Both lanes of the pair (lanes 2k, 2k+1) call it, and both run
// one instruction stream: P[r] is the coupling to the row eliminated before
// (a[r-1] going down, c[r] going up), Q[r] the one towards row m, which the
// elimination overwrites with its reduced value.
// Shuffles and fences name all the warp's calling lanes (`lanes`, the same
// mask on each): with a mask of its own for every pair a warp runs them pair by
// pair, 580 of 1,936 cycles for ten FP64 rows.
template <class T>
__device__ __forceinline__ void thomas_twisted(T *a, const T *b, T *c, T *d, int n, bool top,
                                               unsigned lanes) {
  const int m = n >> 1;
  const int steps = top ? m : n - 1 - m;
  const int dir = top ? 1 : -1;
  const int r0 = top ? 0 : n - 1;
  const T *P = top ? a - 1 : c;
  T *Q = top ? c : a - 1;
  T u = 0, v = 0;  // reduced (Q, d) of the last row eliminated
  // Each row's coefficients are loaded before the stores of the row before
  // (they never overlap), so only the elimination's own chain is serial.
  // The first row has no coupling (pc = 0 leaves b and d as they are).
  int r = r0;
  T pc = 0, bb = 0, qq = 0, dd = 0;
  if (steps > 0) {
    bb = b[r];
    qq = Q[r];
    dd = d[r];
  }
  for (int st = 0; st < steps; ++st) {
    const int rn = r + dir;
    T pcn = 0, bbn = 0, qqn = 0, ddn = 0;
    if (st + 1 < steps) {
      pcn = P[rn];
      bbn = b[rn];
      qqn = Q[rn];
      ddn = d[rn];
    }
    const T ri = recip_t(bb - pc * u);
    u = qq * ri;
    v = (dd - pc * v) * ri;
    Q[r] = u;
    d[r] = v;
    r = rn;
    pc = pcn;
    bb = bbn;
    qq = qqn;
    dd = ddn;
  }
  const T u2 = __shfl_xor_sync(lanes, u, 1), v2 = __shfl_xor_sync(lanes, v, 1);
  const T tu = top ? u : u2, tv = top ? v : v2;  // row m-1: c', d'
  const T bu = top ? u2 : u, bv = top ? v2 : v;  // row m+1: a', d'
  T num = d[m], den = b[m];
  if (m >= 1) {
    num -= a[m - 1] * tv;
    den -= a[m - 1] * tu;
  }
  if (m + 1 <= n - 1) {
    num -= c[m] * bv;
    den -= c[m] * bu;
  }
  T x = num * recip_t(den);
  __syncwarp(lanes);  // both lanes have read row m
  if (top) d[m] = x;
  r = m - dir;
  T qb = 0, db = 0;
  if (steps > 0) {
    qb = Q[r];
    db = d[r];
  }
  for (int st = 0; st < steps; ++st) {
    const int rn = r - dir;
    T qn = 0, dn = 0;
    if (st + 1 < steps) {
      qn = Q[rn];
      dn = d[rn];
    }
    x = db - qb * x;
    d[r] = x;
    r = rn;
    qb = qn;
    db = dn;
  }
}

// Metric determinants of filament q of a block (CalculateBendingForces,
// src/filament.cpp:627-660): det_t forward and det_b backward, each on its
// own lane; filament q's values start at slot (first site) + q.
__device__ __forceinline__ void det_forward(double *sdt, const double *scos, const FilConst &f,
                                            int fb0, int q) {
  const int nn = f.n;
  double *dt = sdt + fb0 + q;
  const double *cs = scos + fb0;
  // The two previous values are carried in registers and each cosine is
  // loaded a row ahead: the recurrence's chain holds no memory access.
  double d2 = 1, d1 = 2;
  dt[0] = d2;
  dt[1] = d1;
  double m = nn > 2 ? -cs[0] : 0.0;
  for (int i = 2; i < nn; ++i) {
    const double mn = i + 1 < nn ? -cs[i - 1] : 0.0;
    const double dn = 2 * d1 - m * m * d2;
    dt[i] = dn;
    d2 = d1;
    d1 = dn;
    m = mn;
  }
}
__device__ __forceinline__ void det_backward(double *sdb, const double *scos, const FilConst &f,
                                             int fb0, int q) {
  const int nn = f.n;
  double *db = sdb + fb0 + q;
  const double *cs = scos + fb0;
  double d2 = 1, d1 = 2;
  db[nn] = d2;
  db[nn - 1] = d1;
  double m = nn > 2 ? -cs[nn - 3] : 0.0;
  for (int i = 2; i < nn; ++i) {
    const double mn = i + 1 < nn ? -cs[nn - i - 2] : 0.0;
    const double dn = 2 * d1 - m * m * d2;
    db[nn - i] = dn;
    d2 = d1;
    d1 = dn;
    m = mn;
  }
}

// v /= |v| over ND components.  Exact: the reference's normalize_vector
// (src/linear_algebra.cpp:26-35).  FAST: one rsqrt and ND products.
template <int ND, bool FAST>
__device__ __forceinline__ double normalize(double *v) {
  double mag = 0.0;
#pragma unroll
  for (int i = 0; i < ND; ++i) mag += v[i] * v[i];
  if (FAST) {
    double inv = rsqrt_nr(mag);
#pragma unroll
    for (int i = 0; i < ND; ++i) v[i] *= inv;
    return mag * inv;
  }
  mag = sqrt(mag);
  bool ok = true;
  const double y = recip_rn(mag, ok);
  double q[ND];
#pragma unroll
  for (int i = 0; i < ND; ++i) q[i] = div_rn(v[i], mag, y, ok);
  if (!ok) {
    asm volatile("" : "+d"(mag));  // a branch: not computed beside the fast path
#pragma unroll
    for (int i = 0; i < ND; ++i) q[i] = v[i] / mag;
  }
#pragma unroll
  for (int i = 0; i < ND; ++i) v[i] = q[i];
  return mag;
}

template <int ND>
__device__ __forceinline__ double dotn(const double *a, const double *b) {
  double m = 0.0;
#pragma unroll
  for (int i = 0; i < ND; ++i) m += a[i] * b[i];
  return m;
}

// Shared-memory words of one integrator block of C sites (the doubles; C/2
// renormalisation flags and the block's filament constants follow).
__host__ __device__ constexpr size_t integrate_smem_doubles(int C) {
  return 28 * (size_t)C;
}

// 8-byte asynchronous global -> shared copy (cp.async), completed by
// cp_async_wait_all() in the same thread.
__device__ __forceinline__ void cp_async8(double *smem_dst, const double *gsrc) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gsrc));
}
__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gsrc) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc));
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::);
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// Block-wide parallel cyclic reduction (Hockney, J. ACM 12:95-113, 1965;
// Hockney & Jesshope, "Parallel Computers 2", 1988, sec. 5.4) of every
// filament's tridiagonal system of the block at once, for the fast
// integrator's blocks of long filaments: the rows laid out as thomas_twisted
// takes them (row i of a filament at slot first + i: lower coefficient in
// a[slot - 1], diagonal b, upper c, right-hand side d).  Each row thread,
// its row scaled to a unit diagonal, eliminates the unknowns s rows away on
// both sides (s = 1, 2, 4, ... below max_rows); a coupling that reaches past
// its filament's rows is zero at every step, so it is skipped.  Rows are
// exchanged through x (3 C) and a, c, d in turn, one barrier a step.  Every
// thread of the block calls it (max_rows is uniform); the solution ends in d.
// O(log n) steps instead of the O(n) sequential elimination, with other
// rounding (the exact integrator keeps the reference's Thomas).  Bound by the
// steps' latency: a step of 256-site blocks took about 620 cycles with two
// barriers and two reciprocals, 470 now.
__device__ __forceinline__ void pcr_block(double *a, const double *b, double *c, double *d,
                                          double *x, int C, bool row, int t, int first, int last,
                                          int max_rows) {
  double lo = 0.0, up = 0.0, rhs = 0.0;
  if (row) {
    const double r = recip_nr(b[t]);
    lo = t > first ? a[t - 1] * r : 0.0;
    up = t < last ? c[t] * r : 0.0;
    rhs = d[t] * r;
  }
  bool mine = false;  // the next exchange goes through a, c, d
  for (int s = 1; s < max_rows; s <<= 1, mine = !mine) {
    double *xl = mine ? a : x, *xu = mine ? c : x + C, *xr = mine ? d : x + 2 * C;
    if (row) {
      xl[t] = lo;
      xu[t] = up;
      xr[t] = rhs;
    }
    __syncthreads();
    if (row) {
      const bool has_m = t - s >= first, has_p = t + s <= last;
      double lm = 0.0, um = 0.0, rm = 0.0, lp = 0.0, upp = 0.0, rp = 0.0;
      if (has_m) {
        lm = xl[t - s];
        um = xu[t - s];
        rm = xr[t - s];
      }
      if (has_p) {
        lp = xl[t + s];
        upp = xu[t + s];
        rp = xr[t + s];
      }
      const double r = recip_nr(fma(-lo, um, fma(-up, lp, 1.0)));
      rhs = fma(-lo, rm, fma(-up, rp, rhs)) * r;
      lo = -(lo * lm) * r;
      up = -(up * upp) * r;
    }
  }
  __syncthreads();  // the last exchange may have read d
  if (row) d[t] = rhs;
}

// Product of two 2 x 2 matrices (row major): c = a b.
__device__ __forceinline__ void mul22(const double a[4], const double b[4], double c[4]) {
  const double c0 = a[0] * b[0] + a[1] * b[2], c1 = a[0] * b[1] + a[1] * b[3];
  const double c2 = a[2] * b[0] + a[3] * b[2], c3 = a[2] * b[1] + a[3] * b[3];
  c[0] = c0;
  c[1] = c1;
  c[2] = c2;
  c[3] = c3;
}

// Metric determinants (CalculateBendingForces, src/filament.cpp:627-660) of a
// fast block's long filaments, as scans of 2 x 2 matrices over the sites:
// joint j takes (x, y) to (2 x - cos^2 y, x), det_t from the tail, det_b from
// the head.  Each warp scans its part of a filament by shuffles; the filament's
// other warps enter through their totals in st (8 doubles a warp).  Joint j's
// thread leaves cos det_t[j] det_b[j + 3] in sg, the last site's 1 / det_t[n - 1]
// in sd[lf].  Every thread of the block calls it; followed by a barrier.  The
// sequential recurrences took 7,100 of a 256-site block's 37,000 cycles, this
// 3,800.
__device__ __forceinline__ void minors_block(bool active, double cosv, int j, int n, int t,
                                             double *st, double *sg, double *sd, int lf) {
  const unsigned FULL = 0xffffffffu;
  const int lane = t & 31, w = t >> 5, base = t - j;
  const bool joint = active && j < n - 2;
  const double c2 = cosv * cosv;
  double P[4] = {1, 0, 0, 1}, B[4];
  if (joint) {
    P[0] = 2;
    P[1] = -c2;
    P[2] = 1;
    P[3] = 0;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) B[i] = P[i];
  for (int s = 1; s < 32; s <<= 1) {
    double q[4], z[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      q[i] = __shfl_up_sync(FULL, P[i], s);
      z[i] = __shfl_down_sync(FULL, B[i], s);
    }
    if (active && j >= s && lane >= s) mul22(P, q, P);
    if (active && j + s < n && lane + s < 32) mul22(B, z, B);
  }
  double e[4], z[4];  // the warp's part before the joint, from either side
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (lane == 31) st[8 * w + i] = P[i];
    if (lane == 0) st[8 * w + 4 + i] = B[i];
    e[i] = __shfl_up_sync(FULL, P[i], 1);
    z[i] = __shfl_down_sync(FULL, B[i], 1);
  }
  __syncthreads();
  if (!active) return;
  double x = 2.0, y = 1.0, p = 2.0, q = 1.0;  // (det_t[1], det_t[0]), (det_b[n-1], det_b[n])
  for (int v = base >> 5; v < w; ++v) {
    const double *m = st + 8 * v;
    const double nx = m[0] * x + m[1] * y;
    y = m[2] * x + m[3] * y;
    x = nx;
  }
  for (int v = (base + n - 1) >> 5; v > w; --v) {
    const double *m = st + 8 * v + 4;
    const double np = m[0] * p + m[1] * q;
    q = m[2] * p + m[3] * q;
    p = np;
  }
  double tx = x, ty = y, bq = q;
  if (lane > 0 && j > 0) {
    tx = e[0] * x + e[1] * y;
    ty = e[2] * x + e[3] * y;
  }
  if (lane < 31 && j + 1 < n) bq = z[2] * p + z[3] * q;
  if (joint) sg[t] = cosv * ty * bq;
  if (j == n - 1) sd[lf] = recip_nr(tx);
}

// MAXC: largest block (sites) the instantiation is launched with; blocks
// per SM requested so that the register budget leaves room for several
// blocks in flight.
template <int MAXC, bool FAST>
struct IntegrateBounds {
  // The exact variant spills below 96 registers; the fast one fits 80, which
  // also holds 4 blocks of 192 sites per SM (2 waves of 17-filament blocks
  // for 20,000 11-site filaments on 148 SMs) and 3 of 256: latency-bound, it
  // gains from the third (20,000 filaments of 5 to 200 bonds, those above 32
  // sites: 303 us a launch with two blocks at 119 registers, 233 with three,
  // for 24 bytes of spills).
  static constexpr int min_blocks =
      MAXC <= 128 ? (FAST ? 6 : 5) : MAXC <= 192 ? (FAST ? 4 : 3) : MAXC <= 256 ? (FAST ? 3 : 2) : 1;
};

// FUSE (fast mixed step only): each bond evaluates its own pairs
// (bond_pair_eval_sum) instead of summing the pair stage's slots.
// FIXC: launched with exactly MAXC threads, so every shared-memory offset is
// a compile-time constant.
template <int ND, int PREC, bool FAST, int MAXC, bool FUSE = false, bool FIXC = false>
__global__ void __launch_bounds__(MAXC, IntegrateBounds<MAXC, FAST>::min_blocks)
    k_integrate(SysConst k, DevState d, int midstep, int rbuf, int interaction,
                int capture) {
  extern __shared__ double smem[];
  const int C = FIXC ? MAXC : (int)blockDim.x;
  double *su = smem;            // site orientations    3C
  double *stn = su + 3 * C;     // tangents             3C
  double *sfr = stn + 3 * C;    // random forces; bond torques in P0-P1  3C
  double *sbF = sfr + 3 * C;    // bond forces, then gamma^-1 F          3C
  double *scos = sbF + 3 * C;   // cos(theta)           C
  double *sT = scos + C;        // rhs / tensions       C
  double *sa = sT + C;          // lower diagonal       C
  double *sb = sa + C;          // diagonal             C
  double *sc = sb + C;          // upper diagonal       C
  double *skeff = sc + C;       // k_eff                C
  double *srp = skeff + C;      // full step: prefetched previous positions 3C
  double *sfp = srp + 3 * C;    // full step: prefetched projected noise     3C
  // New positions (P5 on) take the slots of the previous positions: each
  // thread reads its own previous position before it writes its new one.
  double *sr = srp;             // positions            3C
  // Midstep random forces (P2), read by the projection rows only, before
  // the determinants are written over them.
  double *sfn = sfp;            // 3C
  // The metric determinants (P3): in a midstep in the prefetch area, which
  // only full steps use, so that they are computed alongside the
  // random-force solve; in a full step in the Thomas arrays (sT, sa, sb,
  // sc), free between the two solves' uses.
  double *sdt = midstep ? srp : sT;  // det_t     2C
  double *sdb = sdt + 2 * C;         // det_b     2C
  // The exact step's, where P1's inputs were: det_t and det_b over the bond
  // forces (n + 1 values per filament of at least 3 sites), the tension
  // matrix's elimination (den, inv, up; C each) over the bond torques.  The
  // projection matrix's goes over srp, its solution over sdz.
  double *xdt = sbF, *xdb = sbF + C + C / 2, *xden = sfr;
  double *sdz = sfp + 3 * C;    // full step: prefetched rebuild origin (3C), tracker (C)
  int *sflag = (int *)(sdz + 4 * C);            // C/2 renormalisation flags
  FilConst *sfil = (FilConst *)(sflag + C / 2); // the block's filaments

#define V(arr, slot, comp) arr[(comp) * C + (slot)]

  const int blk = blockIdx.x;
  const int t = threadIdx.x;
  // Without a pair stage in between (fused pairs, or no interactions) the
  // kernel before this one may be the previous integrator step, whose
  // writes every load below reads: wait for it first.
  if (FUSE || !interaction) grid_dep_sync();
  // A rebuild of this step whose list outgrew its segment stops the step
  // before its first store (uniform over the grid: nothing in this kernel
  // sets that bit), so the host can grow the list and redo the step.
  const bool overflowed = (*d.status & ST_HALT) != 0u;
  const unsigned long long mcount = *d.mcount;
  const int un = d.blk_uni_n;
  int s0, count, f0, nfb;
  bool wide = false;
  if (un > 0) {  // equal filaments: the block's range without a table load
    f0 = blk * d.blk_uni_fpb;
    nfb = min(d.blk_uni_fpb, d.nf - f0);
    s0 = f0 * un;
    count = nfb * un;
  } else {
    s0 = d.blk_site0[blk];
    count = d.blk_ns[blk];
    wide = count >= kBlockWide;
    count &= kBlockWide - 1;
    f0 = d.blk_f0[blk];
    nfb = d.blk_nf[blk];
  }
  __shared__ double s_hinv[9];  // the block's system (blocks never mix systems)
  __shared__ uint32_t s_seed;
  // Every global load the step needs is issued here, before the first
  // barrier: the filament constants, the renormalisation state and the
  // block's system constants, below the site state.
  int pre_sw = 0, pre_nn = 0, fid = f0 + t;  // (thread t < nfb) the block's filament t
  if (t < nfb) {
    int slot = 0;
    if (d.blk_slot) {
      const int2 e = d.blk_list[f0 + t];
      fid = e.x;
      slot = e.y;
    }
    sfil[t] = d.fil[fid];
    if (d.blk_slot) sfil[t].site0 = s0 + slot;  // a filament's first slot is site0 - s0
    sflag[t] = 0;
    pre_sw = d.f_switch[fid];
    pre_nn = d.f_nnorm[fid];
  }
  if (t < 10) {
    const int first = d.blk_slot ? d.blk_list[f0].x : f0;
    const ReplicaConst &Rb = d.rep[d.nrep == 1 ? 0 : d.fil[first].rep];
    if (t < 9) s_hinv[t] = Rb.hinv[t];
    else s_seed = Rb.seed;
  }
  const bool active = t < count;
  int g = s0 + t;
  // The site's place in its filament comes from site_jn, so every load of
  // P0 is issued here, alongside the staging of the filament constants,
  // rather than after the barrier.
  int f = 0, lf = 0, jn = 0;
  if (active && un > 0) {
    lf = t / un;
    jn = (t - lf * un) | un << 16;
    f = f0 + lf;
  } else if (active && d.blk_slot) {
    const int4 e = d.blk_slot[(size_t)blk * C + t];
    g = e.x;
    f = e.y;
    jn = e.z;
    lf = e.w;
  } else if (active) {
    f = d.site_fil[g];
    jn = d.site_jn[g];
    lf = f - f0;
  }
  const int n = active ? jn >> 16 : 0;
  const int j = active ? jn & 0xffff : -1;
  const int base = t - j;            // slot of the filament's first site
  const int b = g - f;               // this thread's bond (valid when j < n-1)
  const bool has_bond = active && j < n - 1;

  // ---- P0: positions, orientations, bond forces --------------------------
  double r[3] = {0, 0, 0}, u[3] = {0, 0, 0};
  double bF[3] = {0, 0, 0}, bT[3] = {0, 0, 0};
  int fsw = 0;  // the filament's renormalisation direction before this step
  if (active) {
    fsw = d.f_switch[f];
#pragma unroll
    for (int i = 0; i < ND; ++i) r[i] = d.r[i][g];
    if (!midstep) {
      // The full step needs the midstep's positions and projected noise
      // later; fetch them now, in the background.
      for (int i = 0; i < ND; ++i) cp_async8(&V(srp, t, i), &d.rp[i][g]);
      if (k.stoch)
        for (int i = 0; i < ND; ++i) cp_async8(&V(sfp, t, i), &d.fr[i][g]);
      if (interaction) {  // the displacement tracker's inputs, read last
        for (int i = 0; i < ND; ++i) cp_async8(&V(sdz, t, i), &d.dz[i][g]);
        cp_async8(&V(sdz, t, 3), &d.dt[g]);
      }
      cp_async_commit();
    }
  }
  int e0 = 0, e1 = 0;  // the bond's pair slots
  if (has_bond) {
    // Site orientation = orientation of its bond as Bond::ReInit left it
    // (Mesh::UpdateSiteOrientations, src/mesh.cpp:168-173).
#pragma unroll
    for (int i = 0; i < ND; ++i) u[i] = d.ub[i][b];
    if (!FUSE && interaction) {
      e0 = d.e_off[b];
      e1 = e0 + d.e_cnt[b];
    }
  }
  // Everything above is the previous integrator step's or older; the pair
  // stage just before this kernel writes the bond slots read below.
  grid_dep_sync();
  if (overflowed) {  // uniform over the grid
    cp_async_wait_all();  // no copy into this block's shared memory outlives it
    return;
  }
  if (has_bond && interaction) {
    if (FUSE)
      bond_pair_eval_sum<ND>(k, d, d.rep[d.nrep == 1 ? 0 : d.fil[f].rep].hf, rbuf, b, bF, bT);
    else
      bond_pair_sum<ND, PREC>(d, b, e0, e1, bF, bT);
  }
  if (active && midstep) {  // Mesh::UpdatePrevPositions (src/mesh.cpp:175-182)
#pragma unroll
    for (int i = 0; i < ND; ++i) d.rp[i][g] = r[i];
  }
  if (has_bond) {
    for (int i = 0; i < 3; ++i) {
      V(su, t, i) = u[i];
      V(sbF, t, i) = bF[i];
      V(sfr, t, i) = bT[i];
    }
  }
  __syncthreads();  // the staged filament constants and the bond values
  const FilConst &fc = sfil[active ? lf : 0];  // read from shared memory on use
  // Fast 256-site blocks with a long filament solve by parallel cyclic
  // reduction (uniform over the block).
  int max_rows = 0;
  if (FAST && MAXC > 128)
    for (int q = 0; q < nfb; ++q) max_rows = max(max_rows, sfil[q].n - 1);
  const bool pcr = FAST && MAXC > 128 && (wide || max_rows > kPcrMinRows);
  // First slot of the block's filament q.
  auto slot_of = [&](int q) { return sfil[q].site0 - s0; };
  // Sequential solves of the fast step: from both ends on lanes 2q, 2q+1 (of
  // threads t < 2 nfb: the warp's lanes among them).
  const int pairs_left = 2 * nfb - (t & ~31);
  const unsigned pair_lanes = pairs_left >= 32 ? 0xffffffffu : (1u << max(pairs_left, 0)) - 1u;
  auto solve_rows = [&](int lane_t) {
    if (lane_t < 2 * nfb) {
      const FilConst &f = sfil[lane_t >> 1];
      const int fb0 = slot_of(lane_t >> 1);
      thomas_twisted(sa + fb0, sb + fb0, sc + fb0, sT + fb0, f.n - 1, (lane_t & 1) == 0,
                     pair_lanes);
    }
  };
  // Midstep determinants on warps the random-force solve leaves idle: lanes
  // from g_dt (forward) and g_db (backward), when three warp-aligned groups
  // fit in the block.
  const int g_dt = (2 * nfb + 31) & ~31;
  const int g_db = g_dt + ((nfb + 31) & ~31);
  const bool dets_early = g_db + nfb <= C;
  if (active && j == n - 1) {
    for (int i = 0; i < 3; ++i) u[i] = V(su, t - 1, i);
  }

  // ---- P1: ApplyInteractionForces (src/filament.cpp:992-1048) -------------
  double F[3] = {0.0, 0.0, 0.0};
  if (active) {
    const double mag = 0.5 * 0.0 * fc.l;  // driving_factor 0, from bond centre
    if (j >= 1) {  // this site is site i+1 of bond i = j-1
      double up[3] = {V(su, t - 1, 0), V(su, t - 1, 1), V(su, t - 1, 2)};
      double fb[3] = {V(sbF, t - 1, 0), V(sbF, t - 1, 1), V(sbF, t - 1, 2)};
      double tb[3] = {V(sfr, t - 1, 0), V(sfr, t - 1, 1), V(sfr, t - 1, 2)};
      double pt[3], sf[3];
      cross3(up, tb, pt);
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        pt[i] *= fc.linv;
        sf[i] = 0.5 * fb[i];
      }
#pragma unroll
      for (int i = 0; i < ND; ++i) pt[i] *= -1;
#pragma unroll
      for (int i = 0; i < ND; ++i) F[i] += sf[i];
#pragma unroll
      for (int i = 0; i < ND; ++i) F[i] += pt[i];
#pragma unroll
      for (int i = 0; i < ND; ++i) F[i] += mag * up[i];
    }
    if (j <= n - 2) {  // site i of bond i = j (bF/bT hold this bond)
      double pt[3], sf[3];
      cross3(u, bT, pt);
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        pt[i] *= fc.linv;
        sf[i] = 0.5 * bF[i];
      }
#pragma unroll
      for (int i = 0; i < ND; ++i) F[i] += sf[i];
#pragma unroll
      for (int i = 0; i < ND; ++i) F[i] += pt[i];
#pragma unroll
      for (int i = 0; i < ND; ++i) F[i] += mag * u[i];
    }
  }
  // CalculateAngles (:430-437), CalculateTangents (:439-443, Site::CalcTangent)
  double tn[3] = {0, 0, 0};
  if (active) {
    if (j < n - 2) {
      double un[3] = {V(su, t + 1, 0), V(su, t + 1, 1), V(su, t + 1, 2)};
      scos[t] = dotn<ND>(u, un);
    }
    if (j == 0 || j == n - 1) {
      tn[0] = u[0];
      tn[1] = u[1];
      tn[2] = u[2];
    } else {
#pragma unroll
      for (int i = 0; i < ND; ++i) tn[i] = V(su, t - 1, i) + u[i];
      normalize<ND, FAST>(tn);
    }
    for (int i = 0; i < 3; ++i) V(stn, t, i) = tn[i];
  }
  if (active && j == n - 1) {
    for (int i = 0; i < 3; ++i) V(su, t, i) = u[i];
  }
  // A noisy midstep writes its random forces to the prefetch area (unused in
  // midsteps), not over the bond torques P1 reads, and nothing before its
  // next barrier reads what P1 wrote: only other steps need a barrier here.
  if (!(midstep && k.stoch)) __syncthreads();

  // ---- P2: random forces, projection, previous positions -----------------
  double fr[3] = {0, 0, 0};
  if (midstep && k.stoch && FAST && !pcr) {
    // The mixed step draws, projects and applies its noise in FP32 (its
    // precision contract keeps only the tension solve, the bending forces
    // that feed it and the positions in FP64): the same Philox words, the
    // uniforms to 2^-24, the projection system solved from both ends in FP32
    // over the Thomas arrays' first halves, the projected force added in
    // FP64.
    float *ffn = reinterpret_cast<float *>(sfn);  // 3 x C floats
    float *fT = reinterpret_cast<float *>(sT), *fa = reinterpret_cast<float *>(sa);
    float *fb = reinterpret_cast<float *>(sb), *fcm = reinterpret_cast<float *>(sc);
    float frf[3] = {0.f, 0.f, 0.f};
    const float uf[3] = {(float)u[0], (float)u[1], (float)u[2]};
    if (active) {  // ConstructUnprojectedRandomForces (:518-548)
      uint32_t w[4];
      sc_host_philox4x32_10((uint32_t)j, (uint32_t)mcount, (uint32_t)(mcount >> 32), 0u,
                            s_seed, (uint32_t)fc.f_local, w);
      float xi[3] = {0.f, 0.f, 0.f}, tnf[3] = {0.f, 0.f, 0.f}, txi = 0.f;
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        xi[i] = centered_uniform_f(w[i]);
        tnf[i] = (float)tn[i];
        txi = fmaf(tnf[i], xi[i], txi);
      }
      const float sperp = (float)fc.sperp, dsp = (float)(fc.spar - fc.sperp);
#pragma unroll
      for (int i = 0; i < ND; ++i) frf[i] = fmaf(sperp, xi[i], dsp * txi * tnf[i]);
#pragma unroll
      for (int i = 0; i < ND; ++i) ffn[i * C + t] = frf[i];
    }
    __syncthreads();
    if (has_bond) {  // GeometricallyProjectRandomForces (:550-599)
      float rhs = 0.f;
#pragma unroll
      for (int i = 0; i < ND; ++i) rhs = fmaf(ffn[i * C + t + 1] - frf[i], uf[i], rhs);
      fT[t] = rhs;
      fb[t] = 2.f;
      if (j > 0) {
        fcm[t - 1] = -(float)scos[t - 1];
        fa[t - 1] = -(float)scos[t - 1];
      }
    }
    __syncthreads();
    if (t < 2 * nfb) {
      const FilConst &f = sfil[t >> 1];
      const int fb0 = slot_of(t >> 1);
      thomas_twisted(fa + fb0, fb + fb0, fcm + fb0, fT + fb0, f.n - 1, (t & 1) == 0, pair_lanes);
    }
    if (dets_early) {  // the determinants, on lanes of other warps meanwhile
      if (t >= g_dt && t - g_dt < nfb) det_forward(sdt, scos, sfil[t - g_dt], slot_of(t - g_dt), t - g_dt);
      else if (t >= g_db && t - g_db < nfb) det_backward(sdb, scos, sfil[t - g_db], slot_of(t - g_db), t - g_db);
    }
    __syncthreads();
    if (active) {
      const float tt = j < n - 1 ? fT[t] : 0.f, tp = j > 0 ? fT[t - 1] : 0.f;
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        const float up = j > 0 ? (float)V(su, t - 1, i) : 0.f;
        fr[i] = (double)fmaf(tt, uf[i], fmaf(-tp, up, frf[i]));
      }
#pragma unroll
      for (int i = 0; i < ND; ++i) d.fr[i][g] = fr[i];  // the projected noise, for the full step
    }
  } else if (!FAST) {
    // The exact step: everything that the orientations alone decide -- noise,
    // both matrices' eliminations, the determinants -- then the projection.
    const bool noisy = midstep && k.stoch;
    if (noisy) {
      if (active) {  // ConstructUnprojectedRandomForces (:518-548)
        uint32_t w[4];
        sc_host_philox4x32_10((uint32_t)j, (uint32_t)mcount, (uint32_t)(mcount >> 32), 0u,
                              s_seed, (uint32_t)fc.f_local, w);
        double xi[3] = {0, 0, 0}, xt[3] = {0, 0, 0};
#pragma unroll
        for (int i = 0; i < ND; ++i)
          xi[i] = centered_uniform(w[i]);
        if (ND == 2) {
          xt[0] = tn[0] * tn[0] * xi[0] + tn[0] * tn[1] * xi[1];
          xt[1] = tn[1] * tn[1] * xi[1] + tn[0] * tn[1] * xi[0];
        } else {
          xt[0] = tn[0] * tn[0] * xi[0] + tn[0] * tn[1] * xi[1] +
                  tn[0] * tn[2] * xi[2];
          xt[1] = tn[1] * tn[1] * xi[1] + tn[0] * tn[1] * xi[0] +
                  tn[1] * tn[2] * xi[2];
          xt[2] = tn[2] * tn[2] * xi[2] + tn[0] * tn[2] * xi[0] +
                  tn[1] * tn[2] * xi[1];
        }
#pragma unroll
        for (int i = 0; i < ND; ++i)
          fr[i] = fc.sperp * xi[i] + (fc.spar - fc.sperp) * xt[i];
        for (int i = 0; i < 3; ++i) V(sfn, t, i) = fr[i];
      }
      __syncthreads();
    } else if (!midstep && active) {
      cp_async_wait_all();
      if (k.stoch)
        for (int i = 0; i < ND; ++i) fr[i] = V(sfp, t, i);
    }
    if (has_bond) {
      // Tension matrix (:778-838): it holds no forces.
      double tn2[3] = {V(stn, t + 1, 0), V(stn, t + 1, 1), V(stn, t + 1, 2)};
      const double d1 = dotn<ND>(tn, u), d2 = dotn<ND>(tn2, u);
      sb[t] = fc.two_igperp + fc.dgam * (d1 * d1 + d2 * d2);
      if (j > 0) {
        double u1[3] = {V(su, t - 1, 0), V(su, t - 1, 1), V(su, t - 1, 2)};
        sa[t - 1] = fc.m1_igperp * dotn<ND>(u, u1) - fc.dgam * (dotn<ND>(tn, u1) * d1);
      }
      if (noisy) {  // GeometricallyProjectRandomForces (:550-599)
        double tmp[3];
#pragma unroll
        for (int i = 0; i < ND; ++i) tmp[i] = V(sfn, t + 1, i) - fr[i];
        sT[t] = dotn<ND>(tmp, u);
      }
    }
    __syncthreads();
    if (t < 2 * nfb) {
      const int q = t >> 1, fb0 = slot_of(q);
      const bool trail = (t & 1) != 0;
      double *e = trail ? xden : srp;  // den, inv, up
      factor_and_minors(trail, trail || noisy, scos + fb0, sa + fb0, sb + fb0, e + fb0,
                        e + C + fb0, e + 2 * C + fb0, (trail ? xdb : xdt) + fb0 + q, sfil[q].n);
    }
    __syncthreads();
    if (noisy && t < nfb) {
      const int fb0 = slot_of(t);
      tridiag_rhs<true>(scos + fb0, srp + fb0, srp + C + fb0, srp + 2 * C + fb0, sT + fb0,
                        sdz + fb0, sfil[t].n - 1);
    }
    if (active && j < n - 2) {
      const int dbase = base + lf;
      const double ginv = scos[t] * xdt[dbase + j] * xdb[dbase + j + 3] / xdt[dbase + n - 1];
      skeff[t] = div_by(fc.kappa + fc.l * ginv, fc.l2, fc.l2inv);
    }
    __syncthreads();
    if (noisy && active) {
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        if (j < n - 1) fr[i] = fr[i] + sdz[t] * u[i];
        if (j > 0) fr[i] = fr[i] - sdz[t - 1] * V(su, t - 1, i);
      }
#pragma unroll
      for (int i = 0; i < ND; ++i) d.fr[i][g] = fr[i];  // the projected noise, for the full step
    }
  } else if (midstep) {
    if (k.stoch) {
      if (active) {  // ConstructUnprojectedRandomForces (:518-548)
        uint32_t w[4];
        sc_host_philox4x32_10((uint32_t)j, (uint32_t)mcount, (uint32_t)(mcount >> 32), 0u,
                              s_seed, (uint32_t)fc.f_local, w);
        double xi[3] = {0, 0, 0}, xt[3] = {0, 0, 0};
#pragma unroll
        for (int i = 0; i < ND; ++i)
          xi[i] = centered_uniform(w[i]);
        // (t t^T) xi = (t . xi) t
        const double txi = dotn<ND>(tn, xi);
#pragma unroll
        for (int i = 0; i < ND; ++i) xt[i] = txi * tn[i];
#pragma unroll
        for (int i = 0; i < ND; ++i)
          fr[i] = fc.sperp * xi[i] + (fc.spar - fc.sperp) * xt[i];
        for (int i = 0; i < 3; ++i) V(sfn, t, i) = fr[i];
      }
      __syncthreads();
      // GeometricallyProjectRandomForces (:550-599)
      if (has_bond) {
        double tmp[3];
#pragma unroll
        for (int i = 0; i < ND; ++i) tmp[i] = V(sfn, t + 1, i) - fr[i];
        sT[t] = dotn<ND>(tmp, u);
        sb[t] = 2;
        if (j > 0) {
          sc[t - 1] = -scos[t - 1];
          sa[t - 1] = -scos[t - 1];
        }
      }
      __syncthreads();
      if (pcr) {
        pcr_block(sa, sb, sc, sT, sfr, C, has_bond, t, base, base + n - 2, max_rows);
      } else {
        solve_rows(t);
        if (dets_early) {  // the determinants, on lanes of other warps meanwhile
          if (t >= g_dt && t - g_dt < nfb) det_forward(sdt, scos, sfil[t - g_dt], slot_of(t - g_dt), t - g_dt);
          else if (t >= g_db && t - g_db < nfb) det_backward(sdb, scos, sfil[t - g_db], slot_of(t - g_db), t - g_db);
        }
      }
      __syncthreads();
      if (active) {
        double fp[3];
        if (j == 0) {
#pragma unroll
          for (int i = 0; i < ND; ++i) fp[i] = fr[i] + sT[t] * u[i];
        } else if (j == n - 1) {
#pragma unroll
          for (int i = 0; i < ND; ++i) fp[i] = fr[i] - sT[t - 1] * V(su, t - 1, i);
        } else {
#pragma unroll
          for (int i = 0; i < ND; ++i)
            fp[i] = fr[i] + sT[t] * u[i] - sT[t - 1] * V(su, t - 1, i);
        }
#pragma unroll
        for (int i = 0; i < ND; ++i) fr[i] = fp[i];
#pragma unroll
        for (int i = 0; i < ND; ++i) d.fr[i][g] = fr[i];  // the projected noise, for the full step
      }
    }
  } else if (active) {
    cp_async_wait_all();
    if (k.stoch)
      for (int i = 0; i < ND; ++i) fr[i] = V(sfp, t, i);
  }
  // AddRandomForces (:601-606)
  if (active && k.stoch) {
#pragma unroll
    for (int i = 0; i < ND; ++i) F[i] += fr[i];
  }

  // ---- P3: bending and metric forces (:608-776) ---------------------------
  // (The determinants do not share memory with the projection's solution,
  // which every thread has just read.)
  // (Blocks of long filaments: over srp in midsteps, sT and sa in full ones.)
  double *sdet = midstep ? srp + C : sa;
  if (FAST && pcr) {
    minors_block(active, active && j < n - 2 ? scos[t] : 0.0, j, n, t, midstep ? srp : sT, skeff,
                 sdet, lf);
    __syncthreads();
  } else if (FAST && !(dets_early && midstep && k.stoch)) {
    if (t < nfb) det_forward(sdt, scos, sfil[t], slot_of(t), t);
    else if (t >= C / 2 && t - C / 2 < nfb) det_backward(sdb, scos, sfil[t - C / 2], slot_of(t - C / 2), t - C / 2);
    __syncthreads();
  }
  if (active && FAST) {
    // Each site forms the k_eff of the (up to) three joints its stencil
    // uses from the determinants and cosines, instead of reading them from
    // a barrier later.
    const int dbase = base + lf;
    const double rdet = pcr ? sdet[lf] : recip_nr(sdt[dbase + n - 1]), rl2 = recip_nr(fc.l2);
    auto keff_at = [&](int jj) {
      const double ginv =
          (pcr ? skeff[base + jj] : scos[base + jj] * sdt[dbase + jj] * sdb[dbase + jj + 3]) * rdet;
      return (fc.kappa + fc.l * ginv) * rl2;
    };
    // (I - u2 u2^T) u1 = u1 - (u1 . u2) u2 with the cosines of
    // CalculateAngles: the reference's three stencil terms in vector form.
    double fs[3] = {0, 0, 0};
    const int kk = j;
    if (kk > 1) {
      const double ke = keff_at(j - 2), c = scos[t - 2];
#pragma unroll
      for (int i = 0; i < ND; ++i) fs[i] += ke * (V(su, t - 2, i) - c * V(su, t - 1, i));
    }
    if (kk > 0 && kk < n - 1) {
      const double ke = keff_at(j - 1), c = scos[t - 1];
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        const double um = V(su, t - 1, i);
        fs[i] += ke * ((u[i] - c * um) - (um - c * u[i]));
      }
    }
    if (kk < n - 2) {
      const double ke = keff_at(j), c = scos[t];
#pragma unroll
      for (int i = 0; i < ND; ++i) fs[i] -= ke * (V(su, t + 1, i) - c * u[i]);
    }
#pragma unroll
    for (int i = 0; i < ND; ++i) F[i] += fs[i];
  } else if (active) {
    double fs[3] = {0, 0, 0};
    const int kk = j;
    if (ND == 2) {
      if (kk > 1) {
        double u1[3] = {V(su, t - 2, 0), V(su, t - 2, 1), 0};
        double u2[3] = {V(su, t - 1, 0), V(su, t - 1, 1), 0};
        double ke = skeff[t - 2];
        fs[0] += ke * ((1 - u2[0] * u2[0]) * u1[0] - u2[0] * u2[1] * u1[1]);
        fs[1] += ke * ((1 - u2[1] * u2[1]) * u1[1] - u2[0] * u2[1] * u1[0]);
      }
      if (kk > 0 && kk < n - 1) {
        double u1[3] = {V(su, t - 1, 0), V(su, t - 1, 1), 0};
        double u2[3] = {u[0], u[1], 0};
        double ke = skeff[t - 1];
        fs[0] += ke * ((1 - u1[0] * u1[0]) * u2[0] - u1[0] * u1[1] * u2[1] -
                       ((1 - u2[0] * u2[0]) * u1[0] - u2[0] * u2[1] * u1[1]));
        fs[1] += ke * ((1 - u1[1] * u1[1]) * u2[1] - u1[0] * u1[1] * u2[0] -
                       ((1 - u2[1] * u2[1]) * u1[1] - u2[0] * u2[1] * u1[0]));
      }
      if (kk < n - 2) {
        double u1[3] = {u[0], u[1], 0};
        double u2[3] = {V(su, t + 1, 0), V(su, t + 1, 1), 0};
        double ke = skeff[t];
        fs[0] -= ke * ((1 - u1[0] * u1[0]) * u2[0] - u1[0] * u1[1] * u2[1]);
        fs[1] -= ke * ((1 - u1[1] * u1[1]) * u2[1] - u1[0] * u1[1] * u2[0]);
      }
    } else {
      if (kk > 1) {
        double u1[3] = {V(su, t - 2, 0), V(su, t - 2, 1), V(su, t - 2, 2)};
        double u2[3] = {V(su, t - 1, 0), V(su, t - 1, 1), V(su, t - 1, 2)};
        double ke = skeff[t - 2];
        fs[0] += ke * ((1 - u2[0] * u2[0]) * u1[0] - u2[0] * u2[1] * u1[1] -
                       u2[0] * u2[2] * u1[2]);
        fs[1] += ke * ((1 - u2[1] * u2[1]) * u1[1] - u2[1] * u2[0] * u1[0] -
                       u2[1] * u2[2] * u1[2]);
        fs[2] += ke * ((1 - u2[2] * u2[2]) * u1[2] - u2[2] * u2[0] * u1[0] -
                       u2[2] * u2[1] * u1[1]);
      }
      if (kk > 0 && kk < n - 1) {
        double u1[3] = {V(su, t - 1, 0), V(su, t - 1, 1), V(su, t - 1, 2)};
        const double *u2 = u;
        double ke = skeff[t - 1];
        fs[0] += ke * ((1 - u1[0] * u1[0]) * u2[0] - u1[0] * u1[1] * u2[1] -
                       u1[0] * u1[2] * u2[2] -
                       ((1 - u2[0] * u2[0]) * u1[0] - u2[0] * u2[1] * u1[1] -
                        u2[0] * u2[2] * u1[2]));
        fs[1] += ke * ((1 - u1[1] * u1[1]) * u2[1] - u1[1] * u1[0] * u2[0] -
                       u1[1] * u1[2] * u2[2] -
                       ((1 - u2[1] * u2[1]) * u1[1] - u2[1] * u2[0] * u1[0] -
                        u2[1] * u2[2] * u1[2]));
        fs[2] += ke * ((1 - u1[2] * u1[2]) * u2[2] - u1[2] * u1[0] * u2[0] -
                       u1[2] * u1[1] * u2[1] -
                       ((1 - u2[2] * u2[2]) * u1[2] - u2[2] * u2[0] * u1[0] -
                        u2[1] * u2[2] * u1[1]));
      }
      if (kk < n - 2) {
        const double *u1 = u;
        double u2[3] = {V(su, t + 1, 0), V(su, t + 1, 1), V(su, t + 1, 2)};
        double ke = skeff[t];
        fs[0] -= ke * ((1 - u1[0] * u1[0]) * u2[0] - u1[0] * u1[1] * u2[1] -
                       u1[0] * u1[2] * u2[2]);
        fs[1] -= ke * ((1 - u1[1] * u1[1]) * u2[1] - u1[1] * u1[0] * u2[0] -
                       u1[1] * u1[2] * u2[2]);
        fs[2] -= ke * ((1 - u1[2] * u1[2]) * u2[2] - u1[2] * u1[0] * u2[0] -
                       u1[2] * u1[1] * u2[1]);
      }
    }
#pragma unroll
    for (int i = 0; i < ND; ++i) F[i] += fs[i];
  }

  // ---- P4: tensions (:778-838) --------------------------------------------
  // gamma^-1 = (1/gpar) t t + (1/gperp)(I - t t); the reciprocals are the
  // reference's own quotients 1.0 / friction, computed once per filament.
  auto gam = [&](int a, int c) -> double {
    return fc.igpar * (tn[a] * tn[c]) + fc.igperp * ((a == c ? 1 : 0) - tn[a] * tn[c]);
  };
  // FAST: gamma^-1 F = F / g_perp + (1/g_par - 1/g_perp) (t . F) t
  auto gamF = [&](int i, const double *Fv, double tF) -> double {
    return fc.igperp * Fv[i] + fc.dgam * tF * tn[i];
  };
  if (active) {
    // gamma^-1 F of this site: "temp_a" of row j and "temp_b" of row j-1.
    const double tF = FAST ? dotn<ND>(tn, F) : 0.0;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      double v;
      if (FAST) {
        v = gamF(i, F, tF);
      } else {
        v = gam(i, 0) * F[0] + gam(i, 1) * F[1];
        if (ND == 3) v += gam(i, 2) * F[2];
      }
      V(sbF, t, i) = v;
    }
  }
  __syncthreads();
  if (has_bond) {
    double fdiff[3];
#pragma unroll
    for (int i = 0; i < ND; ++i) fdiff[i] = V(sbF, t + 1, i) - V(sbF, t, i);
    sT[t] = dotn<ND>(u, fdiff);
    if (FAST) {
      double tn2[3] = {V(stn, t + 1, 0), V(stn, t + 1, 1), V(stn, t + 1, 2)};
      double d1 = dotn<ND>(tn, u);
      double d2 = dotn<ND>(tn2, u);
      sb[t] = fc.two_igperp + fc.dgam * (d1 * d1 + d2 * d2);
      if (j > 0) {
        double u1[3] = {V(su, t - 1, 0), V(su, t - 1, 1), V(su, t - 1, 2)};
        double hu = fc.m1_igperp * dotn<ND>(u, u1) -
                    fc.dgam * (dotn<ND>(tn, u1) * dotn<ND>(tn, u));
        sc[t - 1] = hu;
        sa[t - 1] = hu;
      }
    }
  }
  __syncthreads();
  if (!FAST) {
    if (t < nfb) {
      const int fb0 = slot_of(t);
      tridiag_rhs<false>(sa + fb0, xden + fb0, xden + C + fb0, xden + 2 * C + fb0, sT + fb0,
                         sc + fb0, sfil[t].n - 1);
    }
  } else if (pcr) {
    pcr_block(sa, sb, sc, sT, sfr, C, has_bond, t, base, base + n - 2, max_rows);
  } else {
    solve_rows(t);
  }
  __syncthreads();
  const double *sx = FAST ? sT : sc;  // tensions

  // ---- P5: UpdateSitePositions (:840-927), CheckBondLengths (:934-951) ----
  if (active) {
    double fs[3];
    if (j == 0) {
#pragma unroll
      for (int i = 0; i < ND; ++i) fs[i] = sx[t] * u[i];
    } else if (j == n - 1) {
#pragma unroll
      for (int i = 0; i < ND; ++i) fs[i] = -sx[t - 1] * V(su, t - 1, i);
    } else {
#pragma unroll
      for (int i = 0; i < ND; ++i) fs[i] = sx[t] * u[i] - sx[t - 1] * V(su, t - 1, i);
    }
#pragma unroll
    for (int i = 0; i < ND; ++i) F[i] += fs[i];
    const double dl = (midstep ? 0.5 * k.delta : k.delta);
    double rp[3] = {r[0], r[1], r[2]};  // midstep: the previous positions are these
    if (!midstep)
      for (int i = 0; i < ND; ++i) rp[i] = V(srp, t, i);
    const double tF = FAST ? dotn<ND>(tn, F) : 0.0;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      double ft;
      if (FAST) {
        ft = gamF(i, F, tF);
      } else {
        ft = gam(i, 0) * F[0] + gam(i, 1) * F[1];
        if (ND == 3) ft += gam(i, 2) * F[2];
      }
      r[i] = rp[i] + dl * ft;
    }
    for (int i = 0; i < 3; ++i) V(sr, t, i) = r[i];
  }
  __syncthreads();
  double rd[3] = {0, 0, 0}, um = 0.0;
  if (has_bond) {
#pragma unroll
    for (int i = 0; i < ND; ++i) rd[i] = V(sr, t + 1, i) - r[i];
    um = normalize<ND, FAST>(rd);
#pragma unroll
    for (int i = 0; i < ND; ++i) V(su, t, i) = rd[i];
  }
  bool stretched = false;
  if (active && j >= 1) {
    double a = 0.0;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      double temp = r[i] - V(sr, t - 1, i);
      a += temp * temp;
    }
    if (FAST) {
      // |l - |dr|| / l > 1e-3 without the root and the quotient
      const double lo = fc.l * (1.0 - 1e-3), hi = fc.l * (1.0 + 1e-3);
      stretched = a < lo * lo || a > hi * hi;
    } else {
      a = sqrt(a);
      const double err = div_by(dabs(fc.l - a), fc.l, fc.linv);
      stretched = err > 1e-3;
    }
    if (stretched) sflag[lf] = 1;
  }
  // Positions change below only in a block with a filament to renormalise.
  __syncthreads_or(stretched);
  if (t < nfb) {
    int sw = pre_sw, nnorm = pre_nn;
    if (sflag[t]) {
      sw = !sw;
      nnorm = 0;
    }
    nnorm++;
    d.f_switch[fid] = sw;
    d.f_nnorm[fid] = nnorm;
  }
  // The renormalised filament is rebuilt from one end along the bond
  // orientations just computed: from its first site when the switch turns
  // on, else from its last.  Every site runs the chain from that end itself
  // (the same operations in the same order as one sweep over the filament),
  // keeping its own position and its bond's far end, so no site waits for
  // another's result.
  const bool renorm = active && sflag[lf] != 0;
  double rnext[3] = {0, 0, 0};
  if (renorm) {
    const double l = fc.l;
    if (!fsw) {
      double a[3] = {V(sr, base, 0), V(sr, base, 1), V(sr, base, 2)};
      for (int jj = 1; jj <= j; ++jj)
#pragma unroll
        for (int i = 0; i < ND; ++i) a[i] = a[i] + l * V(su, base + jj - 1, i);
      r[0] = a[0];
      r[1] = a[1];
      r[2] = a[2];
      if (j < n - 1) {
        rnext[0] = a[0];
        rnext[1] = a[1];
        rnext[2] = a[2];
#pragma unroll
        for (int i = 0; i < ND; ++i) rnext[i] = a[i] + l * V(su, t, i);
      }
    } else {
      double a[3] = {V(sr, base + n - 1, 0), V(sr, base + n - 1, 1), V(sr, base + n - 1, 2)};
      for (int jj = n - 1; jj > j; --jj) {
        rnext[0] = a[0];
        rnext[1] = a[1];
        rnext[2] = a[2];
#pragma unroll
        for (int i = 0; i < ND; ++i) a[i] = a[i] - l * V(su, base + jj - 1, i);
      }
      r[0] = a[0];
      r[1] = a[1];
      r[2] = a[2];
    }
  }

  // ---- P6: bond geometry (Mesh::UpdateBondPositions), state write-back ----
  double my_dr = 0.0;
  if (active) {
    if (has_bond) {
      // Bond::ReInit on the final sites.  Without renormalisation it repeats
      // the orientation just computed (same operands, same operations).
      double r2[3];
      for (int i = 0; i < 3; ++i) r2[i] = renorm ? rnext[i] : V(sr, t + 1, i);
      double s[3] = {0, 0, 0}, ub[3] = {0, 0, 0}, len, pos[3] = {0, 0, 0}, o[3] = {0, 0, 0};
      if (renorm) {
#pragma unroll
        for (int i = 0; i < ND; ++i) {
          o[i] = r2[i] - r[i];
          ub[i] = o[i];
        }
        len = normalize<ND, FAST>(ub);
      } else {
#pragma unroll
        for (int i = 0; i < ND; ++i) {
          o[i] = r2[i] - r[i];
          ub[i] = rd[i];
        }
        len = um;
      }
#pragma unroll
      for (int i = 0; i < ND; ++i) pos[i] = r[i] + 0.5 * o[i];
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        s[i] = 0.0;
#pragma unroll
        for (int jj = 0; jj < ND; ++jj) s[i] += s_hinv[ND * i + jj] * pos[jj];
        s[i] -= nint(s[i]);
      }
      store_geom<ND>(d, 1 - rbuf, b, s, ub, len, PREC);
#pragma unroll
      for (int i = 0; i < ND; ++i) d.ub[i][b] = ub[i];
    }
#pragma unroll
    for (int i = 0; i < ND; ++i) d.r[i][g] = r[i];
    bool bad = false;
#pragma unroll
    for (int i = 0; i < ND; ++i) bad |= !isfinite(r[i]);
    if (bad) atomicOr(d.status, ST_NAN);
    if (capture) {
      for (int i = 0; i < 3; ++i) d.cap_F[i][g] = F[i];
      if (has_bond) d.cap_T[b] = sx[t];
    }
    // Displacement tracking for the next query (Mesh::UpdateDrTot runs on
    // the filaments whose last update was a full step; each query adds the
    // squared displacement twice, src/mesh.cpp:538-541, src/object.cpp:
    // 282-292).
    if (!midstep && interaction) {
      double acc = V(sdz, t, 3);
      for (int twice = 0; twice < 2; ++twice)
#pragma unroll
        for (int i = 0; i < ND; ++i) {
          double dr = r[i] - V(sdz, t, i);
          acc += dr * dr;
        }
      d.dt[g] = acc;
      my_dr = acc;
    }
  }
  if (!midstep && interaction) {
    // Warp max, then one atomic per warp on the IEEE bits (non-negative),
    // with no barrier.
    double v = my_dr;
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    if ((t & 31) == 0 && v != 0.0) {
      if (!(v <= 1e300)) atomicOr(d.status, ST_NAN);
      atomicMax(&d.dr_max_bits[sfil[0].rep], (unsigned long long)__double_as_longlong(v));
    }
  }
#undef V
}


}  // namespace sc
