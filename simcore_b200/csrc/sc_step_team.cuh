// Integrator of filaments of at most kTeamMaxSites sites: a team of lanes of
// one warp per filament, K consecutive sites a lane.
//
// A warp holds whole filaments back to back (ceil(n / K) lanes each); its
// lanes keep their sites in registers, neighbours are a lane's own sites or
// one shuffle away, and the sequential recurrences run on two lanes per
// filament over a small per-warp shared area, so no block-wide barrier exists.
// Everything that the bond orientations alone decide -- tangents, noise and
// its projection, metric determinants, bending forces, the elimination of
// the tension matrix -- is done before the wait for the pair stage, whose
// forces enter the tension system's right-hand side only.
//
// The arithmetic and its order are those of k_integrate (sc_step.cuh), so the
// exact variant stays bit-identical to the reference
// (src/filament.cpp:394-951, 992-1048).
#pragma once

#include "sc_step.cuh"

namespace sc {

constexpr int kTeamWarps = 4;      // warps per block
constexpr int kTeamMaxFils = 16;   // filaments a warp can hold (two lanes each)

// Shared memory of one warp, in doubles, for S = 32 K site slots.
template <int K>
struct TeamSmem {
  static constexpr int S = 32 * K;
  // Exact: the recurrences' operands.
  static constexpr int cosv = 0;                     // cos(theta) of joint j at its slot
  static constexpr int off = S;                      // tension matrix: coupling of rows j, j + 1
  static constexpr int diag = 2 * S;                 // its diagonal; after its elimination, x
  static constexpr int rhs = 3 * S;                  // right-hand side
  static constexpr int up = 4 * S;                   // eliminated couplings
  static constexpr int den = 5 * S;                  // eliminated diagonal
  static constexpr int inv = 6 * S;                  // its reciprocals
  static constexpr int dett = 7 * S;                 // leading minors, n + 1 per filament
  static constexpr int detb = 8 * S + kTeamMaxFils;  // trailing minors
  // Fast: the coefficients of the reduction (32 each), in their place.
  static constexpr int coef = 0, kCoefs = 20;
  // Renormalisation, after the solves: bond orientations, both end positions
  // of every filament.
  static constexpr int su = off;
  static constexpr int ends = up;
  // Full step: prefetched rp, fr, dz (3 S each) and dt.  Midstep: the
  // projection system (denR, invR, upR, xR; fast: its four FP32 arrays) and,
  // in fr's place, the projected noise.
  static constexpr int pre = 10 * S > 32 * kCoefs ? 10 * S : 32 * kCoefs;
  static constexpr int denR = pre, invR = pre + S, upR = pre + 2 * S, xR = pre + 6 * S;
  static constexpr int fr = pre + 3 * S, dz = pre + 6 * S, dt = pre + 9 * S;
  static constexpr int fil = pre + 10 * S;  // filament constants
  static constexpr int base = fil + kTeamMaxFils * (int)(sizeof(FilConst) / 8);  // first slots
  static constexpr int total = base + kTeamMaxFils / 2;
  static_assert(32 * kCoefs <= pre && detb + S + kTeamMaxFils <= pre && 6 * (32 / ((2 + K) / K)) <= 2 * S && fil % 2 == 0 && total % 2 == 0, "");
};
static_assert(sizeof(FilConst) % 16 == 0, "staged by 16-byte copies");

inline size_t team_smem_bytes(int K) {
  return sizeof(double) * kTeamWarps * (size_t)(K == 1 ? TeamSmem<1>::total : TeamSmem<2>::total);
}

// Sums of the pair slots of a lane's two bonds (bond_pair_sum's, slot by
// slot): consecutive bonds' slots follow one another, so the lane walks one
// run [e0, e0 + c0 + c1) with its loads in batches and changes bonds at
// e0 + c0.
template <int ND, int PREC>
__device__ __forceinline__ void team_pair_sum(const DevState &d, int b0, const bool *bnd, int e0,
                                              int c0, int c1, double F[2][3], double T[2][3]) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
#pragma unroll
    for (int i = 0; i < 3; ++i) F[q][i] = T[q][i] = 0.0;
    if (bnd[q] && d.nx) bond_xlink_sum<ND>(d, b0 + q, F[q], T[q]);
  }
  const int split = e0 + c0, e1 = split + c1;
  if (PREC == 0) {
    constexpr int BATCH = 3;
    const double2 *c = reinterpret_cast<const double2 *>(d.cf64) + 4 * (size_t)e0;
    double a[6] = {F[0][0], F[0][1], F[0][2], T[0][0], T[0][1], T[0][2]};
    for (int e = e0; e < e1; e += BATCH, c += 4 * BATCH) {
      double2 v[BATCH][3];
#pragma unroll
      for (int p = 0; p < BATCH; ++p)
        if (e + p < e1) {
          v[p][0] = c[4 * p];
          v[p][1] = c[4 * p + 1];
          v[p][2] = c[4 * p + 2];
        }
#pragma unroll
      for (int p = 0; p < BATCH; ++p)
        if (e + p < e1) {
          if (e + p == split) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              F[0][i] = a[i];
              T[0][i] = a[3 + i];
              a[i] = F[1][i];
              a[3 + i] = T[1][i];
            }
          }
          a[0] += v[p][0].x;
          a[1] += v[p][0].y;
          if (ND == 3) a[2] += v[p][1].x;
          a[3] += v[p][1].y;
          a[4] += v[p][2].x;
          a[5] += v[p][2].y;
        }
    }
    const int last = c1 > 0 ? 1 : 0;
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (q == last) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          F[q][i] = a[i];
          T[q][i] = a[3 + i];
        }
      }
  } else {
    constexpr int BATCH = 4;
    float sm[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, cm[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const float4 *c = reinterpret_cast<const float4 *>(d.cf32) + 2 * (size_t)e0;
    auto flush = [&](double *Fq, double *Tq) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        Fq[i] += (double)sm[i] - (double)cm[i];
        Tq[i] += (double)sm[3 + i] - (double)cm[3 + i];
        sm[i] = cm[i] = sm[3 + i] = cm[3 + i] = 0.f;
      }
    };
    for (int e = e0; e < e1; e += BATCH, c += 2 * BATCH) {
      float4 v[BATCH][2];
#pragma unroll
      for (int p = 0; p < BATCH; ++p)
        if (e + p < e1) {
          v[p][0] = c[2 * p];
          v[p][1] = c[2 * p + 1];
        }
#pragma unroll
      for (int p = 0; p < BATCH; ++p)
        if (e + p < e1) {
          if (e + p == split) flush(F[0], T[0]);
          kahan_add(sm[0], cm[0], v[p][0].x);
          kahan_add(sm[1], cm[1], v[p][0].y);
          if (ND == 3) kahan_add(sm[2], cm[2], v[p][0].z);
          kahan_add(sm[3], cm[3], v[p][0].w);
          kahan_add(sm[4], cm[4], v[p][1].x);
          kahan_add(sm[5], cm[5], v[p][1].y);
        }
    }
    if (c1 > 0) flush(F[1], T[1]);
    else flush(F[0], T[0]);
  }
}

// FUSE (fast mixed step only): each bond evaluates its own pairs
// (bond_pair_eval_sum) instead of summing the pair stage's slots.
template <int ND, int PREC, bool FAST, int K, bool FUSE = false>
__global__ void __launch_bounds__(kTeamWarps * 32, K == 1 ? 5 : 4)
    k_integrate_team(SysConst k, DevState d, int midstep, int rbuf, int interaction,
                     int capture) {
  static_assert(K == 1 || K == 2, "the lane's sites are written out for one and two");
  using M = TeamSmem<K>;
  constexpr int Q1 = K - 1;  // the lane's last site
  extern __shared__ double team_smem[];
  const unsigned FULL = 0xffffffffu;
  const int t = threadIdx.x & 31;
  const int w = blockIdx.x * kTeamWarps + (threadIdx.x >> 5);
  if (w >= d.n_tm) return;  // whole warps only: nothing below synchronises the block
  // Without a pair stage in between (fused pairs, or no interactions) the
  // kernel before this one may be the previous integrator step, whose
  // writes every load below reads: wait for it first.
  if (FUSE || !interaction) grid_dep_sync();
  double *sm = team_smem + (size_t)(threadIdx.x >> 5) * M::total;
  double *scos = sm + M::cosv, *soff = sm + M::off, *sdiag = sm + M::diag, *srhs = sm + M::rhs;
  double *sdt = sm + M::dett, *sdb = sm + M::detb, *spre = sm + M::pre, *sfr = sm + M::fr;
  const FilConst *sfil = reinterpret_cast<const FilConst *>(sm + M::fil);
  int *sbase = reinterpret_cast<int *>(sm + M::base);
  constexpr int S = M::S;

  // ---- the lane's sites: [j0, j0 + K) of its filament -----------------------
  int f, lf, j0, n, g0, nfw;
  if (d.tm_uni_n > 0) {  // equal filaments: no table load
    const int L = d.tm_uni_lanes, fpw = d.tm_uni_fpw, un = d.tm_uni_n;
    const int f0 = w * fpw;
    nfw = min(fpw, d.nf - f0);
    lf = t / L;
    j0 = (t - lf * L) * K;
    n = lf < nfw ? un : 0;
    if (lf >= nfw) lf = 0;
    f = f0 + lf;
    g0 = f * un + j0;
  } else {
    const int4 q = d.tm_lane[(size_t)w * 32 + t];
    g0 = q.x;
    f = q.y;
    j0 = q.z & 0xffff;
    n = q.z >> 16;
    lf = q.w & 0xff;
    nfw = q.w >> 8;
  }
  const int b0 = g0 - f;         // bond of the lane's first site
  const int slot0 = t * K;       // its slot
  const int sb0 = slot0 - j0;    // slot of the filament's first site
  bool act[K], bnd[K];
#pragma unroll
  for (int q = 0; q < K; ++q) {
    act[q] = j0 + q < n;
    bnd[q] = j0 + q < n - 1;
  }
  const bool lead = act[0] && j0 == 0;

  // ---- every global read of the step, issued together -----------------------
  const bool overflowed = (*d.status & ST_HALT) != 0u;
  const unsigned long long mcount = *d.mcount;
  double r[K][3], u[K][3];
  int e0 = 0, ec[2] = {0, 0};  // the lane's pair slots: first, per bond
  // (The filament constants first: everything below reads them.)
  if (act[0]) {
    constexpr int words = (int)(sizeof(FilConst) / 16);
    for (int i = j0 / K; i < words; i += (n + K - 1) / K)  // by the filament's own lanes
      cp_async16(sm + M::fil + 2 * (words * lf + i),
                 reinterpret_cast<const double2 *>(d.fil + f) + i);
  }
  cp_async_commit();
  if (lead) sbase[lf] = sb0;
#pragma unroll
  for (int q = 0; q < K; ++q) {
#pragma unroll
    for (int i = 0; i < 3; ++i) r[q][i] = u[q][i] = 0.0;
    if (act[q]) {
#pragma unroll
      for (int i = 0; i < ND; ++i) r[q][i] = d.r[i][g0 + q];
    }
    if (bnd[q]) {
#pragma unroll
      for (int i = 0; i < ND; ++i) u[q][i] = d.ub[i][b0 + q];
      if (!FUSE && interaction) {
        if (q == 0) e0 = d.e_off[b0];
        ec[q] = d.e_cnt[b0 + q];
      }
    }
  }
  int fsw = 0, nnorm = 0;  // renormalisation state before this step
  if (act[0]) {
    fsw = d.f_switch[f];
    if (lead) nnorm = d.f_nnorm[f];
  }
  if (!midstep) {
    // The full step needs the midstep's positions and projected noise and
    // the displacement tracker later: fetched in the background.
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (act[q]) {
#pragma unroll
        for (int i = 0; i < ND; ++i) {
          cp_async8(spre + i * S + slot0 + q, &d.rp[i][g0 + q]);
          if (k.stoch) cp_async8(spre + (3 + i) * S + slot0 + q, &d.fr[i][g0 + q]);
          if (interaction) cp_async8(spre + (6 + i) * S + slot0 + q, &d.dz[i][g0 + q]);
        }
        if (interaction) cp_async8(spre + 9 * S + slot0 + q, &d.dt[g0 + q]);
      }
  }
  cp_async_commit();  // (an empty group in midsteps)
  // The system's constants, read late: its box's h^-1 (diagonal), noise key.
  const ReplicaConst &R = d.rep[d.nrep == 1 ? 0 : d.fil[f].rep];
  double hin[3] = {0, 0, 0};
#pragma unroll
  for (int i = 0; i < ND; ++i) hin[i] = R.hinv[(ND + 1) * i];
  const uint32_t seed = R.seed;
  asm volatile("cp.async.wait_group %0;\n" ::"n"(1) : "memory");
  __syncwarp();
  const FilConst &fc = sfil[lf];

  // ---- orientations, angles (:430-437), tangents (:439-443) -----------------
  double um1[3] = {0, 0, 0}, um2[3] = {0, 0, 0}, up1[3] = {0, 0, 0};  // u of sites j0-1, j0-2, j0+K
#pragma unroll
  for (int i = 0; i < ND; ++i) um1[i] = __shfl_up_sync(FULL, u[K - 1][i], 1);
#pragma unroll
  for (int q = 0; q < K; ++q)
    if (act[q] && j0 + q == n - 1) {  // the last site copies the last bond's
#pragma unroll
      for (int i = 0; i < ND; ++i) u[q][i] = q > 0 ? u[q > 0 ? q - 1 : 0][i] : um1[i];
    }
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    um2[i] = K > 1 ? __shfl_up_sync(FULL, u[K > 1 ? K - 2 : 0][i], 1)
                   : __shfl_up_sync(FULL, u[0][i], 2);
    up1[i] = __shfl_down_sync(FULL, u[0][i], 1);
  }
  auto uprev = [&](int q, int i) { return q > 0 ? u[q > 0 ? q - 1 : 0][i] : um1[i]; };
  auto uprev2 = [&](int q, int i) {
    return q > 1 ? u[q > 1 ? q - 2 : 0][i] : q == 1 ? um1[i] : um2[i];
  };
  auto unext = [&](int q, int i) { return q < K - 1 ? u[q < K - 1 ? q + 1 : 0][i] : up1[i]; };
  double cs[K], tn[K][3], tu[K], tm[K];  // cos(theta); tangent; tn . u, tn . u_{j-1}
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const int j = j0 + q;
    cs[q] = tu[q] = tm[q] = 0.0;
    tn[q][0] = tn[q][1] = tn[q][2] = 0.0;
    if (act[q]) {
      if (j < n - 2) {
        double un[3] = {unext(q, 0), unext(q, 1), unext(q, 2)};
        cs[q] = dotn<ND>(u[q], un);
      }
      double um[3] = {uprev(q, 0), uprev(q, 1), uprev(q, 2)};
      if (j == 0 || j == n - 1) {
#pragma unroll
        for (int i = 0; i < ND; ++i) tn[q][i] = u[q][i];
      } else {
#pragma unroll
        for (int i = 0; i < ND; ++i) tn[q][i] = um[i] + u[q][i];
        normalize<ND, FAST>(tn[q]);
      }
      if (j < n - 1) tu[q] = dotn<ND>(tn[q], u[q]);
      if (j > 0) tm[q] = dotn<ND>(tn[q], um);
    }
    if (!FAST) scos[slot0 + q] = cs[q];
  }
  const double csm1 = __shfl_up_sync(FULL, cs[K - 1], 1);
  const double csm2 = K > 1 ? __shfl_up_sync(FULL, cs[K > 1 ? K - 2 : 0], 1)
                            : __shfl_up_sync(FULL, cs[0], 2);
  auto cprev = [&](int q) { return q > 0 ? cs[q > 0 ? q - 1 : 0] : csm1; };
  auto cprev2 = [&](int q) { return q > 1 ? cs[q > 1 ? q - 2 : 0] : q == 1 ? csm1 : csm2; };

  // ---- tension matrix (:778-838): it holds no forces -------------------------
  double dg[K], hu[K];  // row j: diagonal, coupling to row j - 1
  {
    const double tmn = __shfl_down_sync(FULL, tm[0], 1);
#pragma unroll
    for (int q = 0; q < K; ++q) {
      dg[q] = 1.0;
      hu[q] = 0.0;
      if (bnd[q]) {
        const double d1 = tu[q], d2 = q < K - 1 ? tm[q < K - 1 ? q + 1 : 0] : tmn;
        dg[q] = fc.two_igperp + fc.dgam * (d1 * d1 + d2 * d2);
        // (u . u_{j-1} has the bits of cos(theta_{j-1}): the same products.)
        if (j0 + q > 0) hu[q] = fc.m1_igperp * cprev(q) - fc.dgam * (tm[q] * tu[q]);
        if (!FAST) {
          sdiag[slot0 + q] = dg[q];
          if (j0 + q > 0) soff[slot0 + q - 1] = hu[q];
        }
      }
    }
  }

  // ---- noise (midsteps, :518-548) --------------------------------------------
  const bool noisy = midstep && k.stoch;
  double fr[K][3];
  float frf[K][3];
#pragma unroll
  for (int q = 0; q < K; ++q)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      fr[q][i] = 0.0;
      frf[q][i] = 0.f;
    }
  // The mixed step's projection system in FP32.
  float *ffa = reinterpret_cast<float *>(spre), *ffb = ffa + S, *ffc = ffb + S, *ffd = ffc + S;
  if (noisy) {
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (act[q]) {
        uint32_t wv[4];
        sc_host_philox4x32_10((uint32_t)(j0 + q), (uint32_t)mcount, (uint32_t)(mcount >> 32), 0u,
                              seed, (uint32_t)fc.f_local, wv);
        if (FAST) {
          float xi[3] = {0.f, 0.f, 0.f}, tnf[3] = {0.f, 0.f, 0.f}, txi = 0.f;
#pragma unroll
          for (int i = 0; i < ND; ++i) {
            xi[i] = centered_uniform_f(wv[i]);
            tnf[i] = (float)tn[q][i];
            txi = fmaf(tnf[i], xi[i], txi);
          }
          const float sperp = (float)fc.sperp, dsp = (float)(fc.spar - fc.sperp);
#pragma unroll
          for (int i = 0; i < ND; ++i) frf[q][i] = fmaf(sperp, xi[i], dsp * txi * tnf[i]);
        } else {
          double xi[3] = {0, 0, 0}, xt[3] = {0, 0, 0};
          const double *v = tn[q];
#pragma unroll
          for (int i = 0; i < ND; ++i) xi[i] = centered_uniform(wv[i]);
          if (ND == 2) {
            xt[0] = v[0] * v[0] * xi[0] + v[0] * v[1] * xi[1];
            xt[1] = v[1] * v[1] * xi[1] + v[0] * v[1] * xi[0];
          } else {
            xt[0] = v[0] * v[0] * xi[0] + v[0] * v[1] * xi[1] + v[0] * v[2] * xi[2];
            xt[1] = v[1] * v[1] * xi[1] + v[0] * v[1] * xi[0] + v[1] * v[2] * xi[2];
            xt[2] = v[2] * v[2] * xi[2] + v[0] * v[2] * xi[0] + v[1] * v[2] * xi[1];
          }
#pragma unroll
          for (int i = 0; i < ND; ++i) fr[q][i] = fc.sperp * xi[i] + (fc.spar - fc.sperp) * xt[i];
        }
      }
    // Right-hand side of the projection (:550-599).
    double nx[3] = {0, 0, 0};
    float nxf[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      if (FAST) nxf[i] = __shfl_down_sync(FULL, frf[0][i], 1);
      else nx[i] = __shfl_down_sync(FULL, fr[0][i], 1);
    }
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (bnd[q]) {
        if (FAST) {
          float rhs = 0.f;
#pragma unroll
          for (int i = 0; i < ND; ++i)
            rhs = fmaf((q < K - 1 ? frf[q < K - 1 ? q + 1 : 0][i] : nxf[i]) - frf[q][i],
                       (float)u[q][i], rhs);
          ffd[slot0 + q] = rhs;
          ffb[slot0 + q] = 2.f;
          if (j0 + q < n - 2) ffc[slot0 + q] = ffa[slot0 + q] = -(float)cs[q];
        } else {
          double tmp[3];
#pragma unroll
          for (int i = 0; i < ND; ++i)
            tmp[i] = (q < K - 1 ? fr[q < K - 1 ? q + 1 : 0][i] : nx[i]) - fr[q][i];
          srhs[slot0 + q] = dotn<ND>(tmp, u[q]);
        }
      }
  }
  __syncwarp();

  // ---- recurrences of the orientations alone -----------------------------------
  // Two lanes per filament, 2 qf and 2 qf + 1, run the sequential ones.
  const bool odd = (t & 1) != 0;
  const int qf = t >> 1;
  const bool works = qf < nfw;
  const int qb = works ? sbase[qf] : 0, qn = works ? sfil[qf].n : 0;
  double ginv[K] = {};  // metric inverse's element of joint j
  const int li = j0 / K, lanes = (n + K - 1) / K, lane0 = t - li;  // the filament's lanes
  const int lrow = (n - 2) / K;  // its lane with the last row (n = 0: none)
  int nstep = 0;                 // reduction steps of the longest filament of the warp
  if (FAST) {
    const int most = (int)__reduce_max_sync(FULL, (unsigned)lanes);
    while ((1 << nstep) < most) ++nstep;
    // Metric determinants (CalculateBendingForces, :627-660) as scans of 2 x 2
    // matrices over the filament's lanes: joint j takes (x, y) to
    // (2 x - cos^2 y, x), det_t from the tail, det_b from the head.
    const double c0 = cs[0] * cs[0];
    const bool v0 = j0 < n - 2, v1 = K == 2 && j0 + 1 < n - 2;
    double P[4] = {1, 0, 0, 1}, B[4] = {1, 0, 0, 1};
    if (v0) {
      P[0] = B[0] = 2;
      P[1] = B[1] = -c0;
      P[2] = B[2] = 1;
      P[3] = B[3] = 0;
    }
    const double c1 = cs[Q1] * cs[Q1];
    if (v1) {  // both joints of the lane
      P[0] = 4 - c1;
      P[1] = -2 * c0;
      P[2] = 2;
      P[3] = -c0;
      B[0] = 4 - c0;
      B[1] = -2 * c1;
      B[2] = 2;
      B[3] = -c1;
    }
    for (int s = 1; s < most; s <<= 1) {
      double q[4], z[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        q[i] = __shfl_up_sync(FULL, P[i], s);
        z[i] = __shfl_down_sync(FULL, B[i], s);
      }
      if (li >= s) mul22(P, q, P);
      if (li + s < lanes) mul22(B, z, B);
    }
    const double total = 2 * P[0] + P[1];  // det_t past the lane's joints
    const double det_g = __shfl_sync(FULL, total, lane0 + (lanes > 0 ? lanes - 1 : 0));
    double e[4], z[4];  // the scans before the lane's joints
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      e[i] = __shfl_up_sync(FULL, P[i], 1);
      z[i] = __shfl_down_sync(FULL, B[i], 1);
    }
    const bool first = li == 0, last = li + 1 >= lanes;
    const double t0 = first ? 1.0 : 2 * e[2] + e[3], t1 = first ? 2.0 : 2 * e[0] + e[1];
    const double x1 = last ? 2.0 : 2 * z[0] + z[1], y1 = last ? 1.0 : 2 * z[2] + z[3];
    const double rdet = recip_nr(det_g);
    if (v0) ginv[0] = cs[0] * t0 * (v1 ? x1 : y1) * rdet;
    if (v1) ginv[Q1] = cs[Q1] * t1 * y1 * rdet;
    // The tension matrix: with two sites a lane, odd rows eliminated inside
    // the lane; the symmetric system of the (even) rows reduced over the
    // filament's lanes by parallel cyclic reduction (see pcr_block), each
    // step's row scaled to a unit diagonal.  The coefficients stay in shared
    // memory for the right-hand side.
    double *co = sm + M::coef + t;
    double hn = __shfl_down_sync(FULL, hu[0], 1);  // coupling to the next lane's first row
    if (!(j0 + K < n - 1)) hn = 0.0;
    double lo, up, r0;
    if constexpr (K == 2) {
      const double id = recip_nr(dg[Q1]), A = hu[Q1] * id, Bo = hn * id;
      const double pL = Bo * hu[Q1];
      double Bp = __shfl_up_sync(FULL, Bo, 1), Lp = __shfl_up_sync(FULL, pL, 1);
      double Dp = __shfl_up_sync(FULL, Bo * hn, 1);
      if (li == 0) Bp = Lp = Dp = 0.0;
      r0 = recip_nr(dg[0] - Dp - A * hu[Q1]);
      lo = -Lp * r0;
      up = -pL * r0;
      co[0] = id;
      co[32] = A;
      co[64] = Bo;
      co[96] = Bp;
    } else {
      r0 = recip_nr(dg[0]);
      lo = hu[0] * r0;
      up = hn * r0;
    }
    co[128] = r0;
    for (int it = 0; it < nstep; ++it) {
      const int s = 1 << it;
      double lm = __shfl_up_sync(FULL, lo, s), um = __shfl_up_sync(FULL, up, s);
      double lp = __shfl_down_sync(FULL, lo, s), un = __shfl_down_sync(FULL, up, s);
      if (li < s) lm = um = 0.0;
      if (li + s > lrow) lp = un = 0.0;
      const double rr = recip_nr(1.0 - lo * um - up * lp);
      co[32 * (5 + 3 * it)] = lo;
      co[32 * (6 + 3 * it)] = up;
      co[32 * (7 + 3 * it)] = rr;
      lo = -(lo * lm) * rr;
      up = -(up * un) * rr;
    }
    if (noisy && works) {  // the projection system in FP32
      if (!odd) thomas_fast(ffa + qb, ffb + qb, ffc + qb, ffd + qb, qn - 1);
    }
    __syncwarp();
  } else {
    // Lane 2 qf: leading minors det_t, beside the elimination of the
    // projection matrix (midsteps).  Lane 2 qf + 1: trailing minors det_b,
    // beside the elimination of the tension matrix.
    if (works)
      factor_and_minors(odd, odd || noisy, scos + qb, soff + qb, sdiag + qb,
                        sm + (odd ? M::den : M::denR) + qb, sm + (odd ? M::inv : M::invR) + qb,
                        sm + (odd ? M::up : M::upR) + qb, (odd ? sdb : sdt) + qb + qf, qn);
    __syncwarp();
    if (noisy && works && !odd)
      tridiag_rhs<true>(scos + qb, sm + M::denR + qb, sm + M::invR + qb, sm + M::upR + qb,
                        srhs + qb, sm + M::xR + qb, qn - 1);
    if (act[0]) {
      const double det_g = sdt[sb0 + lf + n - 1];
      bool ok = true;
      const double y = recip_rn(det_g, ok);
      double x[K] = {};
#pragma unroll
      for (int q = 0; q < K; ++q)
        if (j0 + q < n - 2) {
          const int db = sb0 + lf + j0 + q;
          x[q] = cs[q] * sdt[db] * sdb[db + 3];
          ginv[q] = div_rn(x[q], det_g, y, ok);
        }
      if (!ok) {
        asm volatile("" : "+d"(x[0]));  // a branch: not computed beside the fast path
#pragma unroll
        for (int q = 0; q < K; ++q)
          if (j0 + q < n - 2) ginv[q] = x[q] / det_g;
      }
    }
    __syncwarp();
  }

  // ---- projected noise, bending and metric forces (:601-776) ------------------
  if (noisy) {
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (act[q]) {
        const int j = j0 + q, s = slot0 + q;
        if (FAST) {
          const float tt = j < n - 1 ? ffd[s] : 0.f, tp = j > 0 ? ffd[s - 1] : 0.f;
#pragma unroll
          for (int i = 0; i < ND; ++i) {
            const float up = j > 0 ? (float)uprev(q, i) : 0.f;
            fr[q][i] = (double)fmaf(tt, (float)u[q][i], fmaf(-tp, up, frf[q][i]));
          }
        } else {
          const double *xR = sm + M::xR + s;
          const double T0 = j < n - 1 ? xR[0] : 0.0, Tm = j > 0 ? xR[-1] : 0.0;
#pragma unroll
          for (int i = 0; i < ND; ++i) {
            if (j < n - 1) fr[q][i] = fr[q][i] + T0 * u[q][i];
            if (j > 0) fr[q][i] = fr[q][i] - Tm * uprev(q, i);
          }
        }
        // Kept where the full step's prefetch puts it.
#pragma unroll
        for (int i = 0; i < ND; ++i) sfr[i * S + s] = fr[q][i];
      }
  }
  double ke[K], fs[K][3];
  {
    const double rl2 = FAST ? recip_nr(fc.l2) : 0.0;
#pragma unroll
    for (int q = 0; q < K; ++q) {
      ke[q] = 0.0;
      if (j0 + q < n - 2) {
        const double x = fc.kappa + fc.l * ginv[q];
        ke[q] = FAST ? x * rl2 : div_by(x, fc.l2, fc.l2inv);
      }
    }
  }
  {
    const double kem1 = __shfl_up_sync(FULL, ke[K - 1], 1);
    const double kem2 = K > 1 ? __shfl_up_sync(FULL, ke[K > 1 ? K - 2 : 0], 1)
                              : __shfl_up_sync(FULL, ke[0], 2);
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const int j = j0 + q;
      const double k1 = q > 0 ? ke[q > 0 ? q - 1 : 0] : kem1;
      const double k2 = q > 1 ? ke[q > 1 ? q - 2 : 0] : q == 1 ? kem1 : kem2;
      fs[q][0] = fs[q][1] = fs[q][2] = 0.0;
      if (!act[q]) continue;
      double um[3] = {uprev(q, 0), uprev(q, 1), uprev(q, 2)};
      double umm[3] = {uprev2(q, 0), uprev2(q, 1), uprev2(q, 2)};
      double un[3] = {unext(q, 0), unext(q, 1), unext(q, 2)};
      double *o = fs[q];
      if (FAST) {
        // (I - u2 u2^T) u1 = u1 - (u1 . u2) u2, with the cosines of
        // CalculateAngles
        const double c1 = cprev(q), c2 = cprev2(q);
        if (j > 1) {
#pragma unroll
          for (int i = 0; i < ND; ++i) o[i] += k2 * (umm[i] - c2 * um[i]);
        }
        if (j > 0 && j < n - 1) {
#pragma unroll
          for (int i = 0; i < ND; ++i)
            o[i] += k1 * ((u[q][i] - c1 * um[i]) - (um[i] - c1 * u[q][i]));
        }
        if (j < n - 2) {
#pragma unroll
          for (int i = 0; i < ND; ++i) o[i] -= ke[q] * (un[i] - cs[q] * u[q][i]);
        }
      } else if (ND == 2) {
        if (j > 1) {
          const double *u1 = umm, *u2 = um;
          o[0] += k2 * ((1 - u2[0] * u2[0]) * u1[0] - u2[0] * u2[1] * u1[1]);
          o[1] += k2 * ((1 - u2[1] * u2[1]) * u1[1] - u2[0] * u2[1] * u1[0]);
        }
        if (j > 0 && j < n - 1) {
          const double *u1 = um, *u2 = u[q];
          o[0] += k1 * ((1 - u1[0] * u1[0]) * u2[0] - u1[0] * u1[1] * u2[1] -
                        ((1 - u2[0] * u2[0]) * u1[0] - u2[0] * u2[1] * u1[1]));
          o[1] += k1 * ((1 - u1[1] * u1[1]) * u2[1] - u1[1] * u1[0] * u2[0] -
                        ((1 - u2[1] * u2[1]) * u1[1] - u2[1] * u2[0] * u1[0]));
        }
        if (j < n - 2) {
          const double *u1 = u[q], *u2 = un;
          o[0] -= ke[q] * ((1 - u1[0] * u1[0]) * u2[0] - u1[0] * u1[1] * u2[1]);
          o[1] -= ke[q] * ((1 - u1[1] * u1[1]) * u2[1] - u1[1] * u1[0] * u2[0]);
        }
      } else {
        if (j > 1) {
          const double *u1 = umm, *u2 = um;
          o[0] += k2 * ((1 - u2[0] * u2[0]) * u1[0] - u2[0] * u2[1] * u1[1] -
                        u2[0] * u2[2] * u1[2]);
          o[1] += k2 * ((1 - u2[1] * u2[1]) * u1[1] - u2[1] * u2[0] * u1[0] -
                        u2[1] * u2[2] * u1[2]);
          o[2] += k2 * ((1 - u2[2] * u2[2]) * u1[2] - u2[2] * u2[0] * u1[0] -
                        u2[2] * u2[1] * u1[1]);
        }
        if (j > 0 && j < n - 1) {
          const double *u1 = um, *u2 = u[q];
          o[0] += k1 * ((1 - u1[0] * u1[0]) * u2[0] - u1[0] * u1[1] * u2[1] -
                        u1[0] * u1[2] * u2[2] -
                        ((1 - u2[0] * u2[0]) * u1[0] - u2[0] * u2[1] * u1[1] -
                         u2[0] * u2[2] * u1[2]));
          o[1] += k1 * ((1 - u1[1] * u1[1]) * u2[1] - u1[1] * u1[0] * u2[0] -
                        u1[1] * u1[2] * u2[2] -
                        ((1 - u2[1] * u2[1]) * u1[1] - u2[1] * u2[0] * u1[0] -
                         u2[1] * u2[2] * u1[2]));
          o[2] += k1 * ((1 - u1[2] * u1[2]) * u2[2] - u1[2] * u1[0] * u2[0] -
                        u1[2] * u1[1] * u2[1] -
                        ((1 - u2[2] * u2[2]) * u1[2] - u2[2] * u2[0] * u1[0] -
                         u2[1] * u2[2] * u1[1]));
        }
        if (j < n - 2) {
          const double *u1 = u[q], *u2 = un;
          o[0] -= ke[q] * ((1 - u1[0] * u1[0]) * u2[0] - u1[0] * u1[1] * u2[1] -
                           u1[0] * u1[2] * u2[2]);
          o[1] -= ke[q] * ((1 - u1[1] * u1[1]) * u2[1] - u1[1] * u1[0] * u2[0] -
                           u1[1] * u1[2] * u2[2]);
          o[2] -= ke[q] * ((1 - u1[2] * u1[2]) * u2[2] - u1[2] * u1[0] * u2[0] -
                           u1[2] * u1[1] * u2[1]);
        }
      }
    }
  }

  // ---- the pair stage's forces (:992-1048) ------------------------------------
  // Everything above is the previous integrator step's or older; the pair
  // stage just before this kernel writes the bond slots read below.
  if (!(FUSE || !interaction)) grid_dep_sync();
  if (overflowed) {       // uniform over the grid
    cp_async_wait_all();  // no copy into this warp's shared memory outlives it
    return;
  }
  if (midstep) {  // Mesh::UpdatePrevPositions (src/mesh.cpp:175-182); the projected noise
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (act[q]) {
#pragma unroll
        for (int i = 0; i < ND; ++i) {
          d.rp[i][g0 + q] = r[q][i];
          if (k.stoch) d.fr[i][g0 + q] = sfr[i * S + slot0 + q];
        }
      }
  }
  double F[K][3];
  {
    double hf[K][3], arm[K][3];  // per bond: half its force, its torque's arm
    double bF[K][3], bT[K][3];
    if (FUSE) {
#pragma unroll
      for (int q = 0; q < K; ++q) {
#pragma unroll
        for (int i = 0; i < 3; ++i) bF[q][i] = bT[q][i] = 0.0;
        if (bnd[q] && interaction) bond_pair_eval_sum<ND>(k, d, R.hf, rbuf, b0 + q, bF[q], bT[q]);
      }
    } else if (interaction) {
      if constexpr (K == 2) {
        team_pair_sum<ND, PREC>(d, b0, bnd, e0, ec[0], ec[1], bF, bT);
      } else if (bnd[0]) {
        bond_pair_sum<ND, PREC>(d, b0, e0, e0 + ec[0], bF[0], bT[0]);
      } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) bF[0][i] = bT[0][i] = 0.0;
      }
    } else {
#pragma unroll
      for (int q = 0; q < K; ++q)
#pragma unroll
        for (int i = 0; i < 3; ++i) bF[q][i] = bT[q][i] = 0.0;
    }
#pragma unroll
    for (int q = 0; q < K; ++q) {
      cross3(u[q], bT[q], arm[q]);
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        arm[q][i] *= fc.linv;
        hf[q][i] = 0.5 * bF[q][i];
      }
    }
    double hm[3] = {0, 0, 0}, am[3] = {0, 0, 0};
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      hm[i] = __shfl_up_sync(FULL, hf[K - 1][i], 1);
      am[i] = __shfl_up_sync(FULL, arm[K - 1][i], 1);
    }
    if (!midstep) cp_async_wait_all();
#pragma unroll
    for (int q = 0; q < K; ++q) {
      const int j = j0 + q;
      F[q][0] = F[q][1] = F[q][2] = 0.0;
      if (!act[q]) continue;
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        double x = 0.0;
        if (j >= 1) {
          x += q > 0 ? hf[q > 0 ? q - 1 : 0][i] : hm[i];
          x -= q > 0 ? arm[q > 0 ? q - 1 : 0][i] : am[i];
        }
        if (j <= n - 2) {
          x += hf[q][i];
          x += arm[q][i];
        }
        if (k.stoch) x += sfr[i * S + slot0 + q];
        x += fs[q][i];
        F[q][i] = x;
      }
    }
  }

  // ---- tensions (:778-838) -----------------------------------------------------
  // gamma^-1 = (1/gpar) t t + (1/gperp)(I - t t)
  auto gamma_inv_F = [&](int q, double out[3]) {
    const double *v = tn[q], *x = F[q];
    if (FAST) {
      const double tF = dotn<ND>(v, x);
#pragma unroll
      for (int i = 0; i < ND; ++i) out[i] = fc.igperp * x[i] + fc.dgam * tF * v[i];
    } else {
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        double s = 0.0;
#pragma unroll
        for (int c = 0; c < ND; ++c) {
          const double g = fc.igpar * (v[i] * v[c]) +
                           fc.igperp * ((i == c ? 1 : 0) - v[i] * v[c]);
          if (c == 0) s = g * x[0];
          else s += g * x[c];
        }
        out[i] = s;
      }
    }
  };
  double ten[K] = {};  // right-hand side, then tension of bond j
  {
    double gF[K][3], gn[3] = {0, 0, 0};
#pragma unroll
    for (int q = 0; q < K; ++q) {
      gF[q][0] = gF[q][1] = gF[q][2] = 0.0;
      if (act[q]) gamma_inv_F(q, gF[q]);
    }
#pragma unroll
    for (int i = 0; i < ND; ++i) gn[i] = __shfl_down_sync(FULL, gF[0][i], 1);
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (bnd[q]) {
        double fd[3];
#pragma unroll
        for (int i = 0; i < ND; ++i)
          fd[i] = (q < K - 1 ? gF[q < K - 1 ? q + 1 : 0][i] : gn[i]) - gF[q][i];
        ten[q] = dotn<ND>(u[q], fd);
      }
  }
  double tenm = 0.0;  // of bond j0 - 1
  if (FAST) {
    const double *co = sm + M::coef + t;
    double x = ten[0];
    if constexpr (K == 2) {
      double rp = __shfl_up_sync(FULL, ten[Q1], 1);
      if (li == 0) rp = 0.0;
      x = x - co[96] * rp - co[32] * ten[Q1];
    }
    x *= co[128];
    for (int it = 0; it < nstep; ++it) {
      const int s = 1 << it;
      const double lo = co[32 * (5 + 3 * it)], up = co[32 * (6 + 3 * it)];
      const double rr = co[32 * (7 + 3 * it)];
      double xm = __shfl_up_sync(FULL, x, s), xp = __shfl_down_sync(FULL, x, s);
      if (li < s) xm = 0.0;
      if (li + s > lrow) xp = 0.0;
      x = (x - lo * xm - up * xp) * rr;
    }
    ten[0] = bnd[0] ? x : 0.0;
    if constexpr (K == 2) {
      double xn = __shfl_down_sync(FULL, x, 1);
      if (li + 1 > lrow) xn = 0.0;
      ten[Q1] = bnd[Q1] ? ten[Q1] * co[0] - co[32] * x - co[64] * xn : 0.0;
    }
    tenm = __shfl_up_sync(FULL, ten[Q1], 1);
  } else {
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (bnd[q]) srhs[slot0 + q] = ten[q];
    __syncwarp();
    if (works && !odd)
      tridiag_rhs<false>(soff + qb, sm + M::den + qb, sm + M::inv + qb, sm + M::up + qb,
                         srhs + qb, sdiag + qb, qn - 1);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < K; ++q)
      if (bnd[q]) ten[q] = sdiag[slot0 + q];
    if (act[0] && j0 > 0) tenm = sdiag[slot0 - 1];
  }

  // ---- UpdateSitePositions (:840-927), CheckBondLengths (:934-951) -------------
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const int j = j0 + q, s = slot0 + q;
    if (!act[q]) continue;
    const double T0 = ten[q], Tm = q > 0 ? ten[q > 0 ? q - 1 : 0] : tenm;
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      double x;
      if (j == 0) x = T0 * u[q][i];
      else if (j == n - 1) x = -Tm * uprev(q, i);
      else x = T0 * u[q][i] - Tm * uprev(q, i);
      F[q][i] += x;
    }
    const double dl = midstep ? 0.5 * k.delta : k.delta;
    double ft[3] = {0, 0, 0};
    gamma_inv_F(q, ft);
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      const double rp = midstep ? r[q][i] : spre[i * S + s];
      r[q][i] = rp + dl * ft[i];
    }
  }
  double rn[3] = {0, 0, 0};
#pragma unroll
  for (int i = 0; i < ND; ++i) rn[i] = __shfl_down_sync(FULL, r[0][i], 1);
  double rd[K][3], len[K];
  bool bad = false;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    len[q] = 0.0;
    rd[q][0] = rd[q][1] = rd[q][2] = 0.0;
    if (bnd[q]) {
      double m2 = 0.0;
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        rd[q][i] = (q < K - 1 ? r[q < K - 1 ? q + 1 : 0][i] : rn[i]) - r[q][i];
        m2 += rd[q][i] * rd[q][i];
      }
      len[q] = normalize<ND, FAST>(rd[q]);
      if (FAST) {
        // |l - |dr|| / l > 1e-3 without the root and the quotient
        const double lo = fc.l * (1.0 - 1e-3), hi = fc.l * (1.0 + 1e-3);
        bad = bad || m2 < lo * lo || m2 > hi * hi;
      } else {
        bad = bad || div_by(dabs(fc.l - len[q]), fc.l, fc.linv) > 1e-3;
      }
    }
  }
  const unsigned bad_lanes = __ballot_sync(FULL, bad);
  const unsigned fil_lanes =
      act[0] ? (unsigned)((((unsigned long long)1 << lanes) - 1ull) << lane0) : 0u;
  const bool renorm = (bad_lanes & fil_lanes) != 0u;
  if (lead) {
    d.f_switch[f] = renorm ? !fsw : fsw;
    d.f_nnorm[f] = renorm ? 1 : nnorm + 1;
  }
  if (bad_lanes != 0u) {
    // The renormalised filament is rebuilt from one end along the bond
    // orientations just computed: from its first site when the switch turns
    // on, else from its last.  Every lane runs the chain from that end to its
    // own sites (the operations of one sweep, in its order).
    double *su = sm + M::su, *ends = sm + M::ends + 6 * lf;
#pragma unroll
    for (int q = 0; q < K; ++q) {
      if (bnd[q]) {
#pragma unroll
        for (int i = 0; i < ND; ++i) su[i * S + slot0 + q] = rd[q][i];
      }
      if (act[q] && j0 + q == 0) {
#pragma unroll
        for (int i = 0; i < ND; ++i) ends[i] = r[q][i];
      }
      if (act[q] && j0 + q == n - 1) {
#pragma unroll
        for (int i = 0; i < ND; ++i) ends[3 + i] = r[q][i];
      }
    }
    __syncwarp();
    if (act[0] && renorm) {
      const double l = fc.l;
      double a[3] = {0, 0, 0};
      if (!fsw) {
#pragma unroll
        for (int i = 0; i < ND; ++i) a[i] = ends[i];
#pragma unroll 4
        for (int jj = 0; jj < j0; ++jj)
#pragma unroll
          for (int i = 0; i < ND; ++i) a[i] = a[i] + l * su[i * S + sb0 + jj];
#pragma unroll
        for (int q = 0; q < K; ++q)
          if (act[q]) {
#pragma unroll
            for (int i = 0; i < ND; ++i) {
              r[q][i] = a[i];
              if (bnd[q]) a[i] = a[i] + l * rd[q][i];
            }
          }
      } else {
#pragma unroll
        for (int i = 0; i < ND; ++i) a[i] = ends[3 + i];
        const int jl = min(j0 + K, n);  // past the lane's last site
#pragma unroll 4
        for (int jj = n - 1; jj >= jl; --jj)
#pragma unroll
          for (int i = 0; i < ND; ++i) a[i] = a[i] - l * su[i * S + sb0 + jj - 1];
        // a is site jl - 1's position; each bond leads to the one before.
#pragma unroll
        for (int q = K - 1; q >= 0; --q)
          if (act[q]) {
            if (j0 + q < jl - 1) {
#pragma unroll
              for (int i = 0; i < ND; ++i) a[i] = a[i] - l * rd[q][i];
            }
#pragma unroll
            for (int i = 0; i < ND; ++i) r[q][i] = a[i];
          }
      }
    }
  }

  // ---- bond geometry (Mesh::UpdateBondPositions), state write-back -------------
#pragma unroll
  for (int i = 0; i < ND; ++i) rn[i] = __shfl_down_sync(FULL, r[0][i], 1);
  double my_dr = 0.0;
  bool nan = false;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const int g = g0 + q, b = b0 + q, s = slot0 + q;
    if (bnd[q]) {
      // Bond::ReInit on the final sites; without renormalisation it repeats
      // the orientation just computed (same operands, same operations).
      double sp[3] = {0, 0, 0}, ub[3] = {0, 0, 0}, ln = len[q];
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        const double o = (q < K - 1 ? r[q < K - 1 ? q + 1 : 0][i] : rn[i]) - r[q][i];
        ub[i] = renorm ? o : rd[q][i];
        // h^-1 is diagonal: the other products are zeros.
        sp[i] = hin[i] * (r[q][i] + 0.5 * o);
        sp[i] -= nint(sp[i]);
      }
      if (renorm) ln = normalize<ND, FAST>(ub);
      store_geom<ND>(d, 1 - rbuf, b, sp, ub, ln, PREC);
#pragma unroll
      for (int i = 0; i < ND; ++i) d.ub[i][b] = ub[i];
    }
    if (act[q]) {
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        d.r[i][g] = r[q][i];
        nan |= !isfinite(r[q][i]);
      }
      if (capture) {
        for (int i = 0; i < 3; ++i) d.cap_F[i][g] = F[q][i];
        if (bnd[q]) d.cap_T[b] = ten[q];
      }
      // Displacement tracking for the next rebuild check: each query adds the
      // squared displacement twice (src/mesh.cpp:538-541, src/object.cpp:282-292).
      if (!midstep && interaction) {
        double acc = spre[9 * S + s];
        for (int twice = 0; twice < 2; ++twice)
#pragma unroll
          for (int i = 0; i < ND; ++i) {
            const double dr = r[q][i] - spre[(6 + i) * S + s];
            acc += dr * dr;
          }
        d.dt[g] = acc;
        my_dr = fmax(my_dr, acc);
        nan |= !(acc <= 1e300);
      }
    }
  }
  if (nan) atomicOr(d.status, ST_NAN);
  if (!midstep && interaction) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) my_dr = fmax(my_dr, __shfl_xor_sync(FULL, my_dr, o));
    if (t == 0) {
      // Non-negative doubles order as their bit patterns; most warps see a
      // larger maximum already and skip the atomic.
      const unsigned long long bits = (unsigned long long)__double_as_longlong(my_dr);
      unsigned long long *slot = &d.dr_max_bits[fc.rep];
      if (bits > *(volatile unsigned long long *)slot) atomicMax(slot, bits);
    }
  }
}

}  // namespace sc
