// Device building blocks of the fused batched evaluation of valence, Coulomb + Lennard-Jones and
// Generalized Born terms, shared by the evaluation kernel and the minimization kernel.
//
// One thread block evaluates one work unit at a time: a group of whole molecules whose atoms
// fit in shared memory.  Everything a molecule needs stays on chip for the whole evaluation:
//
//   stage       int64 fixed-point coordinates -> (hi, lo) float pairs, per-atom parameters,
//               per-molecule Lennard-Jones tables
//   valence     bonds, angles, dihedrals and their attached 1-4 pairs
//               (Potential/valence_potential.tpp:9-1420 restated for FP32)
//   GB pass 1   Born-radius descreening sums psi_i over all pairs, both directions
//               (Potential/nonbonded_potential.tpp:511-728)
//   radii       effective radii, GB self energy and its dE/dR (nonbonded_potential.tpp:730-805)
//   pass 2      Coulomb + Lennard-Jones on non-excluded pairs, GB pair energy and force, dE/dR
//               sums (nonbonded_potential.tpp:8-425, 808-975)
//   chain rule  OBC prefactor on dE/dR (nonbonded_potential.tpp:982-1021)
//   pass 3      radius chain-rule forces (nonbonded_potential.tpp:1022-1290)
//   commit      forces into the int64 + int32-overflow arrays, energies into per-system slots
//
// Pair passes walk 32 x 32 tiles of a molecule's lower triangle, one tile per warp, two pairs per
// lane and step in packed FP32 (FFMA2 and kin).  A block's 32 atoms are held as 16 records of two
// atoms q and q + 16; lane l holds atom i in registers, meets record (l + k) mod 16 at step k, and
// the accumulators of a record's two j atoms travel with it through the 16 lanes of the half warp
// (walkTile).  A tile whose block I has at most 16 atoms takes half the steps, both half warps
// holding those atoms.  Forces, psi and dE/dR leave registers once per tile through integer
// shared-memory atomics, so every sum is independent of scheduling and the results are
// bit-identical run to run.
//
// What bounds the passes is instruction issue.  Against one pair a lane and step from 16-byte
// records per atom, the packed form issues about half the FP32 instructions per pair, and a half
// warp reads 16 records of 16 bytes where 32 lanes read 32: half the shared-memory wavefronts.
// With the branch-free descreening of hctSeries2: 1,024 molecules of 16-256 atoms, force + energy
// with its copies, 445 -> 391 us; 60 minimization cycles of 4,096 molecules of 24-96 atoms 61.5 ->
// 50.7 ms; 32 chains of 2,000-5,000 atoms 1,817 -> 1,600 us.
//
// Shared memory per atom pair record: pa = (x, x', y, y'), pb = (z, z', w1, w1'), pc = (lo x, lo
// x', lo y, lo y'), pd = (lo z, lo z', w2, w2') and pg = (g, g', h, h'), where w1 / w2 carry what
// the pass needs (pass 1 and 3: s*rho and rho; pass 2: charge and effective radius), g the
// reciprocal effective radius and h the Lennard-Jones code bits (pass 2) or the chain-rule dE/dR
// (pass 3). prm holds the static per-atom values.
#ifndef STORMM_B200_UNIT_EVAL_CUH
#define STORMM_B200_UNIT_EVAL_CUH

#include <cuda_runtime.h>

#include <mutex>
#include <set>
#include <utility>

#include "device_kits.h"
#include "fixed_point.cuh"

namespace sb {

namespace {

// Constants/generalized_born.h:21-44 (Taylor series of the HCT integral at long range)
constexpr float kTaylorA = 0.33333333333333333333f;
constexpr float kTaylorB = 0.4f;
constexpr float kTaylorC = 0.42857142857142857143f;
constexpr float kTaylorD = 0.44444444444444444444f;
constexpr float kTaylorDD = 0.45454545454545454545f;
constexpr float kTaylorE = 1.33333333333333333333f;
constexpr float kTaylorF = 2.4f;
constexpr float kTaylorG = 3.42857142857142857143f;
constexpr float kTaylorH = 4.44444444444444444444f;
constexpr float kTaylorHH = 5.45454545454545454545f;

constexpr unsigned kFullMask = 0xffffffffu;

// ------------------------------------------------------------------------------------------------
// Clash damping: softened Coulomb and Lennard-Jones cores (Potential/soft_core_potentials.tpp:
// 30-52 and 140-180, as the clash-forgiving GPU kernels apply them,
// nonbonded_potential_tilegroups.cui:536-602)
// ------------------------------------------------------------------------------------------------
// Clash distance and sigma ratio of a molecule in minimization cycle `cycle` of a damping over
// `cycles` cycles (both shrink linearly to zero, hpc_minimization.cu:268-272); cycle < 0: the
// base values unscaled
__device__ __forceinline__ float2 clashScaled(float distance, float ratio, int cycles, int cycle) {
  if (cycle < 0) {
    return make_float2(distance, ratio);
  }
  if (cycle >= cycles) {
    return make_float2(0.0f, 0.0f);
  }
  const double progress = static_cast<double>(cycles - cycle) / static_cast<double>(cycles);
  return make_float2(static_cast<float>(static_cast<double>(distance) * progress),
                     static_cast<float>(static_cast<double>(ratio) * progress));
}

// Constants of the quadratic Coulomb core for a clash distance cd > 0: below cd the pair energy
// is qiqj (a (r + 1)^2 + b), continuous in value and slope with qiqj / r at cd
__device__ __forceinline__ float2 quadraticCore(float cd) {
  if (cd <= 0.0f) {
    return make_float2(0.0f, 0.0f);
  }
  const float a = -0.5f / (cd * cd * (cd + 1.0f));
  return make_float2(a, 1.0f / cd - a * (cd + 1.0f) * (cd + 1.0f));
}

// Coulomb and Lennard-Jones terms of one pair with softened cores: the quadratic Coulomb core
// (constants qc from quadraticCore) below the clash distance cd, the quartic Lennard-Jones core
// below ratio x sigma, sigma = (A / B)^(1/6) (none where B <= 1e-6).  Adds the energies to
// *e_elec and *e_vdw and returns the force factor (force on j = factor x (r_j - r_i)).
__device__ __forceinline__ float softCorePair(float r, float invr, float qiqj, float lja,
                                              float ljb, float cd, float2 qc, float ratio,
                                              float* e_elec, float* e_vdw) {
  float fmag;
  if (r < cd) {
    const float rp = r + 1.0f;
    *e_elec = __fadd_rn(*e_elec, __fmul_rn(qiqj, fmaf(qc.x * rp, rp, qc.y)));
    fmag = (r > 1.0e-10f) ? qiqj * (2.0f * qc.x + 2.0f * qc.x * invr) : 0.0f;
  }
  else {
    *e_elec = __fadd_rn(*e_elec, __fmul_rn(qiqj, invr));
    fmag = -(qiqj * invr * invr * invr);
  }
  const float rl = (ljb > 1.0e-6f) ? ratio * sqrtf(cbrtf(__fdividef(lja, ljb))) : 0.0f;
  if (r < rl) {
    const float il = 1.0f / rl;
    const float il2 = il * il;
    const float il6 = il2 * il2 * il2;
    const float a = ((6.0f * ljb - 12.0f * lja * il6) * il * il6) /
                    (((4.0f * rl + 12.0f) * rl + 12.0f) * rl + 4.0f);
    const float rlp = rl + 1.0f;
    const float rlp2 = rlp * rlp;
    const float b = (lja * il6 - ljb) * il6 - a * rlp2 * rlp2;
    const float rp = r + 1.0f;
    const float a3 = a * rp * rp * rp;
    *e_vdw = __fadd_rn(*e_vdw, fmaf(a3, rp, b));
    if (r > 1.0e-10f) {
      fmag += 4.0f * a3 * invr;
    }
  }
  else {
    const float invr2 = invr * invr;
    const float invr4 = invr2 * invr2;
    *e_vdw = __fadd_rn(*e_vdw, __fmul_rn(__fsub_rn(__fmul_rn(__fmul_rn(lja, invr4), invr4),
                                                   __fmul_rn(ljb, invr2)), invr4));
    fmag += (6.0f * ljb - 12.0f * lja * invr4 * invr2) * invr4 * invr4;
  }
  return fmag;
}

// Valence geometry in FP64 (the angle, dihedral and 1-4 terms of both precision modes)
__device__ __forceinline__ double3 sub3d(double3 a, double3 b) {
  return make_double3(a.x - b.x, a.y - b.y, a.z - b.z);
}
__device__ __forceinline__ double dot3d(double3 a, double3 b) {
  return fma(a.x, b.x, fma(a.y, b.y, a.z * b.z));
}
__device__ __forceinline__ double3 cross3d(double3 a, double3 b) {
  return make_double3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// valence_potential.tpp: below this squared cosine between consecutive dihedral bonds the force
// divides by the sine squared; above it (near-collinear atoms) it takes the fixed reciprocal
constexpr double kAsymptoticToOne = 0.99999904632568359375;
constexpr double kInvOneMinusAsymptote = 1048576.0;

// Softened cores in FP64 (Potential/soft_core_potentials.tpp:30-52, 140-180; softCorePair in
// double)
// Quadratic Coulomb core below cd: qiqj (a (r + 1)^2 + b), continuous in value and slope
__device__ __forceinline__ double2 quadraticCore64(double cd) {
  if (cd <= 0.0) {
    return make_double2(0.0, 0.0);
  }
  const double a = -0.5 / (cd * cd * (cd + 1.0));
  return make_double2(a, 1.0 / cd - a * (cd + 1.0) * (cd + 1.0));
}

// Coulomb and Lennard-Jones energies of one pair with softened cores added to *e_elec, *e_vdw;
// returns the force factor (force on j = factor x (r_j - r_i))
__device__ __forceinline__ double softCorePair64(double r, double invr, double qiqj, double lja,
                                                 double ljb, double cd, double2 qc, double ratio,
                                                 double* e_elec, double* e_vdw) {
  double fmag;
  if (r < cd) {
    const double rp = r + 1.0;
    *e_elec += qiqj * (qc.x * rp * rp + qc.y);
    fmag = (r > 1.0e-10) ? qiqj * (2.0 * qc.x + 2.0 * qc.x * invr) : 0.0;
  }
  else {
    *e_elec += qiqj * invr;
    fmag = -(qiqj * invr * invr * invr);
  }
  const double rl = (ljb > 1.0e-6) ? ratio * pow(lja / ljb, 1.0 / 6.0) : 0.0;
  if (r < rl) {
    const double il = 1.0 / rl;
    const double il2 = il * il;
    const double il6 = il2 * il2 * il2;
    const double a = ((6.0 * ljb - 12.0 * lja * il6) * il * il6) /
                     (((4.0 * rl + 12.0) * rl + 12.0) * rl + 4.0);
    const double rlp = rl + 1.0;
    const double rlp2 = rlp * rlp;
    const double b = (lja * il6 - ljb) * il6 - a * rlp2 * rlp2;
    const double rp = r + 1.0;
    const double a3 = a * rp * rp * rp;
    *e_vdw += a3 * rp + b;
    if (r > 1.0e-10) {
      fmag += 4.0 * a3 * invr;
    }
  }
  else {
    const double invr2 = invr * invr;
    const double invr4 = invr2 * invr2;
    *e_vdw += (lja * invr4 * invr4 - ljb * invr2) * invr4;
    fmag += (6.0 * ljb - 12.0 * lja * invr4 * invr2) * invr4 * invr4;
  }
  return fmag;
}


// Packed FP32 pairs (Blackwell FFMA2 / FADD2 / FMUL2): two pairs of one lane in one instruction
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.0f), a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }


// HCT descreening of an atom of offset radius rho by a neighbour of screened radius sj at
// distance r (invr = 1/r): the amounts psi decreases by, and their radial derivative factors
// -(1/r) dI/dr, for two pairs at once in packed FP32.
//
// Beyond r = 4 sj the reference's Taylor series applies (nonbonded_potential.tpp:590-596,
// 1116-1121): with t = (sj / r)^2, the first five terms of
//   I = (sj t / r^2) sum_k k / (2k + 1) t^(k-1),
//   -(1/r) dI/dr = (sj t / r^4) sum_k k (2k + 2) / (2k + 1) t^(k-1).
// Closer in, while the spheres do not overlap (r > rho + sj), the reference's closed form
// (:597-604, :1122-1128) is the same series summed to infinity.  hctSeries2 takes both: five
// terms, plus t^5 times a polynomial in t for the rest of the series where r <= 4 sj (weighted
// minimax fits on 1/16 <= t <= 0.3: relative error of the sums below 1.1e-8 and 4.3e-9).  No
// reciprocal, logarithm or cancellation, so it is more accurate than the closed form in FP32.
// It tells where it does not apply (overlapping spheres, or t > 0.3): bonded neighbours mostly, a
// few pairs per atom, which hctClosed2 evaluates after the tile's walk (spreadLate), in place of
// a branch per step on r <= 4 sj, which nearly every step of a small molecule takes on some lane
// (with each lane evaluating its own such pairs in turn, the busiest lane, with some eight, set the
// cost and the gain was 1 %).
// BRANCH: the polynomial behind a branch, for tiles where most steps have no pair within 4 sj.
// FAR: every pair is known to lie beyond 4 sj and apart.
constexpr float kSeriesLimit = 0.3f;

struct Near2 {
  bool x, y;
};

template <bool DERIV, bool BRANCH, bool FAR = false>
__device__ __forceinline__ Near2 hctSeries2(float2 r, float2 invr, float2 rho, float2 sj,
                                            float2* integral, float2* deriv) {
  const float2 invr2 = mul2(invr, invr);
  const float2 t = mul2(mul2(sj, sj), invr2);
  const float2 touch = add2(rho, sj);
  const bool near_x = t.x > 0.0625f;
  const bool near_y = t.y > 0.0625f;
  float2 ti = f2(0.0f), td = f2(0.0f);
  if (!FAR && (!BRANCH || near_x || near_y)) {
    ti = fma2(t, f2(1.4148261547e0f), f2(7.0001393557e-2f));
    ti = fma2(t, ti, f2(5.3365993500e-1f));
    ti = fma2(t, ti, f2(4.5760014653e-1f));
    ti = f2(near_x ? ti.x : 0.0f, near_y ? ti.y : 0.0f);
    if (DERIV) {
      td = fma2(t, f2(4.3931625366e1f), f2(-9.4689912796e0f));
      td = fma2(t, td, f2(1.3106045723e1f));
      td = fma2(t, td, f2(6.9396967888e0f));
      td = fma2(t, td, f2(6.4842333794e0f));
      td = f2(near_x ? td.x : 0.0f, near_y ? td.y : 0.0f);
    }
  }
  ti = FAR ? f2(kTaylorDD) : fma2(t, ti, f2(kTaylorDD));
  ti = fma2(t, ti, f2(kTaylorD));
  ti = fma2(t, ti, f2(kTaylorC));
  ti = fma2(t, ti, f2(kTaylorB));
  ti = fma2(t, ti, f2(kTaylorA));
  const float2 scale = mul2(mul2(sj, t), invr2);
  *integral = mul2(scale, ti);
  if (DERIV) {
    td = FAR ? f2(kTaylorHH) : fma2(t, td, f2(kTaylorHH));
    td = fma2(t, td, f2(kTaylorH));
    td = fma2(t, td, f2(kTaylorG));
    td = fma2(t, td, f2(kTaylorF));
    td = fma2(t, td, f2(kTaylorE));
    *deriv = mul2(mul2(scale, invr2), td);
  }
  if (FAR) {
    return Near2{false, false};
  }
  // written so that a distance that is not a number (r = 0) is left to the closed forms, which add
  // nothing there
  return Near2{!(r.x > touch.x && t.x <= kSeriesLimit), !(r.y > touch.y && t.y <= kSeriesLimit)};
}

// The same from the closed forms, for both directions of one pair at any distance.  The three the
// reference selects by overlap case
// (no overlap, partial overlap, atom inside the neighbour's sphere: nonbonded_potential.tpp:
// 597-628) are one expression in U = r + sj and L = max(rho, |r - sj|):
//   I = 1/2 [1/L - 1/U + (sj^2 - r^2)/(4r) (1/L^2 - 1/U^2) + ln(L/U) / (2r)]
//       + (1/rho - 1/L) when rho < sj - r,
// and I = 0 when rho >= U.  Its derivative (:1129-1165), lambda = dL/dr being 1 without overlap, 0
// on partial overlap and -1 inside the neighbour, q = (sj^2 - r^2)/(4r) and q' = dq/dr:
//   dI/dr = 1/2 [-lambda/L^2 + 1/U^2 + q'(1/L^2 - 1/U^2) + 2q (1/U^3 - lambda/L^3)
//                + (lambda/L - 1/U - ln(L/U)/r) / (2r)] - 1/L^2 (inside).
// Returns (I.x, I.y, derivative factor .x, .y).  ln(L / U) needs an accurate absolute
// value where the form cancels: the fast hardware logarithm (__logf) errs by about 1e-7 absolute
// with a consistent sign, which biased every atom's psi by -6.5e-7 relative and the GB energy by
// +1.1e-6 relative (1,024 molecules of 16-256 atoms); logf removes the bias.
template <bool DERIV>
__device__ __forceinline__ float4 hctClosed2(float r, float r2, float invr, float2 rho, float2 sj) {
  const float invr2 = invr * invr;
  const bool far_x = r > 4.0f * sj.x;
  const bool far_y = r > 4.0f * sj.y;
  const float2 sj2 = mul2(sj, sj);
  float2 vfi = f2(0.0f), vfd = f2(0.0f), vnd = f2(0.0f);
  if (far_x || far_y) {
    const float2 t = mul2(sj2, f2(invr2));
    float2 di = fma2(t, f2(kTaylorDD), f2(kTaylorD));
    di = fma2(t, di, f2(kTaylorC));
    di = fma2(t, di, f2(kTaylorB));
    di = fma2(t, di, f2(kTaylorA));
    const float2 tsr = mul2(mul2(sj, t), f2(invr2));
    vfi = mul2(tsr, di);
    if (DERIV) {
      float2 dd = fma2(t, f2(kTaylorHH), f2(kTaylorH));
      dd = fma2(t, dd, f2(kTaylorG));
      dd = fma2(t, dd, f2(kTaylorF));
      dd = fma2(t, dd, f2(kTaylorE));
      vfd = mul2(mul2(tsr, f2(invr2)), dd);
    }
  }
  const float2 u = add2(f2(r), sj);
  const float2 rms = sub2(f2(r), sj);
  const float2 l = f2(fmaxf(rho.x, fabsf(rms.x)), fmaxf(rho.y, fabsf(rms.y)));
  const bool in_x = -rms.x > rho.x;      // inside the neighbour's sphere
  const bool in_y = -rms.y > rho.y;
  const float2 lu = mul2(l, u);
  const float2 inv_lu = f2(__fdividef(1.0f, lu.x), __fdividef(1.0f, lu.y));
  const float2 il = mul2(u, inv_lu);
  const float2 iu = mul2(l, inv_lu);
  const float2 liu = mul2(l, iu);
  const float2 lg = f2(logf(liu.x), logf(liu.y));
  const float2 s2mr2 = sub2(sj2, f2(r2));
  // the integral
  const float2 dlu = sub2(il, iu);
  const float2 q = mul2(mul2(f2(0.25f * invr), s2mr2), dlu);
  float2 v = add2(fma2(q, add2(il, iu), dlu), mul2(f2(0.5f * invr), lg));
  if (in_x) {
    v.x += 2.0f * (__fdividef(1.0f, rho.x) - il.x);
  }
  if (in_y) {
    v.y += 2.0f * (__fdividef(1.0f, rho.y) - il.y);
  }
  const float2 vni = f2((rho.x < u.x) ? 0.5f * v.x : 0.0f, (rho.y < u.y) ? 0.5f * v.y : 0.0f);
  if (DERIV) {
    // its derivative, lambda = dL/dr
    const float2 lam = f2((rms.x >= rho.x) ? 1.0f : (in_x ? -1.0f : 0.0f),
                          (rms.y >= rho.y) ? 1.0f : (in_y ? -1.0f : 0.0f));
    const float2 il2 = mul2(il, il);
    const float2 iu2 = mul2(iu, iu);
    const float2 q2 = mul2(f2(0.5f * invr), s2mr2);
    const float2 dq = mul2(f2(-0.25f), fma2(sj2, f2(invr2), f2(1.0f)));
    const float2 lil2 = mul2(lam, il2);
    float2 dv = sub2(iu2, lil2);
    dv = fma2(dq, sub2(il2, iu2), dv);
    dv = fma2(q2, sub2(mul2(iu2, iu), mul2(lil2, il)), dv);
    dv = fma2(f2(0.5f * invr), sub2(sub2(mul2(lam, il), iu), mul2(f2(invr), lg)), dv);
    dv = sub2(mul2(f2(0.5f), dv), f2(in_x ? il2.x : 0.0f, in_y ? il2.y : 0.0f));
    const float2 w = mul2(dv, f2(-invr));
    vnd = f2((rho.x < u.x) ? w.x : 0.0f, (rho.y < u.y) ? w.y : 0.0f);
  }
  return make_float4(far_x ? vfi.x : vni.x, far_y ? vfi.y : vni.y, far_x ? vfd.x : vnd.x,
                     far_y ? vfd.y : vnd.y);
}

// Neck GB (Mongan's neck between two spheres, nonbonded_potential.tpp:678-702, 1219-1245): pairs
// closer than rho_i + rho_j + 2 offset + cutoff add scale * V / (1 + m^2 + 0.3 m^6), m = r - S,
// to the descreening, with V and S looked up for the pair's neck indices
struct NeckGb {
  const float* sep;
  const float* val;
  int size;
  float scale;
  float reach;     // 2 offset + cutoff: the pair takes the neck term when r < rho_i + rho_j + reach
  __device__ explicit NeckGb(const DevSynthesis &d) :
      sep(d.neck_sep), val(d.neck_val), size(d.neck_size), scale(d.neck_scale),
      reach(2.0f * d.gb_offset + d.neck_cut) {}
  // the amount psi of the atom with index ni decreases by from the atom with index nj
  __device__ __forceinline__ float integral(int ni, int nj, float r) const {
    const int t = size * nj + ni;
    const float m = r - __ldg(&sep[t]);
    const float m2 = m * m;
    return __fdividef(scale * __ldg(&val[t]), 1.0f + m2 + 0.3f * m2 * m2 * m2);
  }
  // the same and its radial derivative factor -(1/r) dI/dr
  __device__ __forceinline__ float both(int ni, int nj, float r, float invr, float* deriv) const {
    const int t = size * nj + ni;
    const float m = r - __ldg(&sep[t]);
    const float m2 = m * m;
    const float v = scale * __ldg(&val[t]);
    const float inv_den = __fdividef(1.0f, 1.0f + m2 + 0.3f * m2 * m2 * m2);
    *deriv = (2.0f * m + 1.8f * m2 * m2 * m) * v * inv_den * inv_den * invr;
    return v * inv_den;
  }
};

// Shared-memory layout of one work unit
struct UnitSmem {
  float4* pa;       // x, y (hi parts) of the record's two atoms
  float4* pb;       // z (hi), pass payload w1
  float4* pc;       // x, y (lo parts)
  float4* pd;       // z (lo), pass payload w2
  float4* pg;       // 1 / effective radius; Lennard-Jones code bits in pass 2, dE/dR after the
                    // chain rule
  float4* prm;      // charge * sqrt(k_Coulomb), Lennard-Jones code (int bits), rho, s * rho
  int* fx;          // int63 force accumulators: primary
  int* fy;
  int* fz;
  int* fxo;         // overflow
  int* fyo;
  int* fzo;
  int* psi;         // int63 psi accumulator, 2^kPsiBits
  int* psio;
  int* de;          // int63 dE/dR accumulator, 2^kDeijdaBits
  int* deo;
  int* neck;        // neck GB table index of the atom
  float2* lj;       // Lennard-Jones tables of the unit's molecules
  unsigned long long* nrg;   // per unit molecule energies
  int* meta;        // the unit's rows of DevSynthesis::unit_meta by field: metaStride entries each,
  int metaStride;   // one per molecule and the closing one
  int* sys;         // molecule index, number of atoms, first slot: views into meta
  int* natom;
  int* slot0;
  float2* clash;    // per unit molecule: clash distance and sigma ratio of this evaluation
  unsigned short* late;   // kLateEntries per warp: pairs of GB pass 1 set aside (RadiiPass)
};

// Field f of unit molecule k's row (k = number of molecules: the closing row)
__device__ __forceinline__ int unitMeta(const UnitSmem &s, int f, int k) {
  return s.meta[f * s.metaStride + k];
}

// Atom pair records: slot s of a unit is atom (s / 16) % 2 of record 16 (s / 32) + s % 16
constexpr int kRecords = kTile / 2;
__device__ __forceinline__ int slotRecord(int slot) {
  return (slot >> 5) * kRecords + (slot & (kRecords - 1));
}
__device__ __forceinline__ int slotHalf(int slot) { return (slot >> 4) & 1; }
// Component c (0: first pair, 2: second pair) of a slot in a record array
__device__ __forceinline__ float &slotValue(float4* a, int slot, int c) {
  return reinterpret_cast<float*>(a)[4 * slotRecord(slot) + c + slotHalf(slot)];
}

__host__ __device__ inline size_t alignUp(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Raise a kernel's dynamic shared-memory limit to the device's opt-in maximum, once per kernel and
// device (the attribute belongs to the function on the current device); launches then pass only
// their own size, and the per-system drop-in, a launch per molecule, pays no attribute call
template <class K>
cudaError_t allowLargeSmem(K kern) {
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> done;
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_pair(reinterpret_cast<const void*>(kern), dev);
  if (done.count(key) != 0) return cudaSuccess;
  int optin = 0;
  err = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (err != cudaSuccess) return err;
  // static and dynamic shared memory together may not exceed the opt-in maximum
  cudaFuncAttributes attr;
  err = cudaFuncGetAttributes(&attr, kern);
  if (err != cudaSuccess) return err;
  err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin - static_cast<int>(attr.sharedSizeBytes));
  if (err == cudaSuccess) {
    done.insert(key);
  }
  else {
    cudaGetLastError();   // reported here, not left for the next launch check to find
  }
  return err;
}

constexpr int kSlotBytes = 5 * 8 + 16 + 11 * 4;
constexpr int kLateEntries = 128;   // per warp: pairs of a tile set aside before they are evaluated

// Most molecules a work unit of max_slots atom slots can hold (each takes at least a tile's edge)
__host__ __device__ inline int unitSystems(int max_slots) {
  const int n = max_slots / kTile;
  return n < kMaxUnitSystems ? n : kMaxUnitSystems;
}

// Dynamic shared memory of one work unit's evaluation by a block of `threads`: max_slots atom
// slots, max_lj table entries
__host__ __device__ inline size_t unitSmemBytes(int max_slots, int max_lj, int threads) {
  const int max_sys = unitSystems(max_slots);
  size_t b = static_cast<size_t>(kSlotBytes) * max_slots;
  b = alignUp(b, 16);
  b += sizeof(float2) * max_lj;
  b = alignUp(b, 16);
  b += sizeof(unsigned long long) * max_sys * kNrgStride;
  b += sizeof(float2) * max_sys;
  b += sizeof(int) * kUnitMetaFields * (max_sys + 1);
  b += sizeof(unsigned short) * kLateEntries * (threads / 32);
  return alignUp(b, 16);
}

__device__ UnitSmem carveSmem(char* base, int max_slots, int max_lj) {
  const int max_sys = unitSystems(max_slots);
  UnitSmem s;
  size_t off = 0;
  const size_t records = sizeof(float4) * (max_slots / 2);
  s.pa = reinterpret_cast<float4*>(base + off); off += records;
  s.pb = reinterpret_cast<float4*>(base + off); off += records;
  s.pc = reinterpret_cast<float4*>(base + off); off += records;
  s.pd = reinterpret_cast<float4*>(base + off); off += records;
  s.pg = reinterpret_cast<float4*>(base + off); off += records;
  s.prm = reinterpret_cast<float4*>(base + off); off += sizeof(float4) * max_slots;
  int* ip = reinterpret_cast<int*>(base + off);
  s.fx = ip; ip += max_slots;
  s.fy = ip; ip += max_slots;
  s.fz = ip; ip += max_slots;
  s.fxo = ip; ip += max_slots;
  s.fyo = ip; ip += max_slots;
  s.fzo = ip; ip += max_slots;
  s.psi = ip; ip += max_slots;
  s.psio = ip; ip += max_slots;
  s.de = ip; ip += max_slots;
  s.deo = ip; ip += max_slots;
  s.neck = ip; ip += max_slots;
  off = alignUp(off + 11 * sizeof(int) * max_slots, 16);
  s.lj = reinterpret_cast<float2*>(base + off); off += sizeof(float2) * max_lj;
  off = alignUp(off, 16);
  s.nrg = reinterpret_cast<unsigned long long*>(base + off);
  off += sizeof(unsigned long long) * max_sys * kNrgStride;
  s.clash = reinterpret_cast<float2*>(base + off);
  off += sizeof(float2) * max_sys;
  int* q = reinterpret_cast<int*>(base + off);
  s.meta = q;
  s.metaStride = max_sys + 1;
  s.sys = q + kMetaSystem * (max_sys + 1);
  s.natom = q + kMetaAtoms * (max_sys + 1);
  s.slot0 = q + kMetaSlot * (max_sys + 1);
  q += kUnitMetaFields * (max_sys + 1);
  s.late = reinterpret_cast<unsigned short*>(q);
  return s;
}

// The threads that evaluate one work unit together: a whole block
struct BlockTeam {
  __device__ __forceinline__ int rank() const { return threadIdx.x; }
  __device__ __forceinline__ int size() const { return blockDim.x; }
  __device__ __forceinline__ int warp() const { return threadIdx.x >> 5; }
  __device__ __forceinline__ int warps() const { return blockDim.x >> 5; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
  __device__ __forceinline__ bool any(bool p) const { return __syncthreads_or(p) != 0; }
};

// Index of the unit molecule that owns position pos of a prefix-sum array of n + 1 entries
__device__ __forceinline__ int findOwner(const int* prefix, int n, int pos) {
  int k = 0;
  while (k + 1 < n && prefix[k + 1] <= pos) {
    k++;
  }
  return k;
}

// Tile (I, J), I >= J, of the lower triangle from its index within the molecule
__device__ __forceinline__ void tileCoordinates(int local, int* ti, int* tj) {
  int i = static_cast<int>((sqrtf(8.0f * local + 1.0f) - 1.0f) * 0.5f);
  while (i * (i + 1) / 2 > local) i--;
  while ((i + 1) * (i + 2) / 2 <= local) i++;
  *ti = i;
  *tj = local - i * (i + 1) / 2;
}

// High and low parts of a slot's coordinates
__device__ __forceinline__ float3 slotHi(const UnitSmem &s, int slot) {
  return make_float3(slotValue(s.pa, slot, 0), slotValue(s.pa, slot, 2), slotValue(s.pb, slot, 0));
}
__device__ __forceinline__ float3 slotLo(const UnitSmem &s, int slot) {
  return make_float3(slotValue(s.pc, slot, 0), slotValue(s.pc, slot, 2), slotValue(s.pd, slot, 0));
}

// Coordinate difference b - a from the hi / lo representation of two slots
__device__ __forceinline__ float3 slotDelta(const UnitSmem &s, int a, int b) {
  const float3 ah = slotHi(s, a), al = slotLo(s, a), bh = slotHi(s, b), bl = slotLo(s, b);
  return make_float3((bh.x - ah.x) + (bl.x - al.x), (bh.y - ah.y) + (bl.y - al.y),
                     (bh.z - ah.z) + (bl.z - al.z));
}

__device__ __forceinline__ void addForce(const UnitSmem &s, int slot, float fx, float fy, float fz,
                                         float scale) {
  atomicAddInt63(fx * scale, &s.fx[slot], &s.fxo[slot]);
  atomicAddInt63(fy * scale, &s.fy[slot], &s.fyo[slot]);
  atomicAddInt63(fz * scale, &s.fz[slot], &s.fzo[slot]);
}

// Warp-wide int64 sum, result in every lane
__device__ __forceinline__ long long warpSum(long long v) {
  for (int o = 16; o > 0; o >>= 1) {
    v += __shfl_xor_sync(kFullMask, v, o);
  }
  return v;
}

// A tile's energy in the output fixed-point format: the lanes' FP64 sums added by an xor
// butterfly (every lane adds the same two values at every level, so all lanes hold the same bits
// and the total does not depend on which warp ran the tile), then rounded once.  Rounding each
// lane's share instead loses the pairs of distant tiles, whose per-lane sums fall below one unit
// of 2^-26 kcal/mol (1.6e-6 of the Lennard-Jones energy of a 2,100-atom chain), and an integer
// accumulator finer than the output overflows on clashing starting structures (1.6e7 kcal/mol).
__device__ __forceinline__ long long tileEnergy(double v, float nrg_scale) {
  for (int o = 16; o > 0; o >>= 1) {
    v += __shfl_xor_sync(kFullMask, v, o);
  }
  return __double2ll_rn(v * static_cast<double>(nrg_scale));
}

// Warp-reduce one scaled energy per lane (all lanes in one molecule) into its slot
__device__ __forceinline__ void warpEnergy(const UnitSmem &s, int k, int slot, float e,
                                           float scale) {
  const long long v = warpSum(__float2ll_rn(e * scale));
  if ((threadIdx.x & 31) == 0 && v != 0) {
    atomicAdd(&s.nrg[k * kNrgStride + slot], static_cast<unsigned long long>(v));
  }
}

// ------------------------------------------------------------------------------------------------
// Valence terms (Potential/valence_potential.tpp).  Warps take chunks of 32 terms of one molecule,
// so each chunk's energies reduce across the warp into a single shared-memory update.
// ------------------------------------------------------------------------------------------------
// The three kinds of valence terms, taken in chunks of 32 that never straddle two molecules
enum ValenceKind : int { kBondTerms = 0, kAnglTerms, kDiheTerms };

// A lane's term of a chunk: its molecule, its index in the synthesis' list, and whether the chunk
// reaches this lane
struct ValenceTerm {
  int k;
  int index;
  bool valid;
};

// First item of a list for rank r of n that take it in turn, when `before` items of other lists
// have been dealt out before it: the ranks that took one item less come first
__device__ __forceinline__ int dealFrom(int r, int n, int before) {
  const int v = (r - before) % n;
  return v < 0 ? v + n : v;
}

// Where valence terms read their atoms and put forces and energies: a work unit's shared memory.
// The chunks of the three kinds are dealt to the warps in one sequence, as are the GB tiles after
// them, so that a small molecule's dihedrals, angles, bonds and tiles run on different warps side
// by side and not on the first warps one after another (with the molecule table of a unit read in
// one step: 60 minimization cycles of one 48-atom molecule 6.20 -> 5.18 ms, 384 molecules of 20-200
// atoms 165 -> 159 us).
struct SmemValence {
  const UnitSmem &s;
  int nsys;
  int rank;
  int stride;
  __device__ SmemValence(const UnitSmem &s_in, int nsys_in, int rank_in, int stride_in) :
      s(s_in), nsys(nsys_in), rank(rank_in), stride(stride_in) {}
  __device__ __forceinline__ int chunks(int kind) const {
    return unitMeta(s, kMetaBondChunk + kind, nsys);
  }
  __device__ __forceinline__ int begin(int before) const { return dealFrom(rank, stride, before); }
  __device__ __forceinline__ int chunkStride() const { return stride; }
  __device__ __forceinline__ ValenceTerm term(int kind, int c, int lane) const {
    const int* first = s.meta + (kMetaBondChunk + kind) * s.metaStride;
    const int k = findOwner(first, nsys, c);
    const int rel = c - first[k];
    const int tail = (unitMeta(s, kMetaTypes, k) >> (8 + 6 * kind)) & 63;
    const int here = (c + 1 == first[k + 1]) ? tail : 32;
    return ValenceTerm{k, unitMeta(s, kMetaBond0 + kind, k) + 32 * rel + lane, lane < here};
  }
  __device__ __forceinline__ int slot0(int k) const { return s.slot0[k]; }
  __device__ __forceinline__ float3 hi(int i) const { return slotHi(s, i); }
  __device__ __forceinline__ float3 lo(int i) const { return slotLo(s, i); }
  __device__ __forceinline__ void force(int i, float fx, float fy, float fz, float scale) const {
    addForce(s, i, fx, fy, fz, scale);
  }
  __device__ __forceinline__ void energy(int k, int slot, float e, float scale) const {
    warpEnergy(s, k, slot, e, scale);
  }
  // exact coordinates of a slot: the hi + lo float pair summed in double
  __device__ __forceinline__ double3 pos64(int i) const {
    const float3 a = slotHi(s, i);
    const float3 b = slotLo(s, i);
    return make_double3(static_cast<double>(a.x) + static_cast<double>(b.x),
                        static_cast<double>(a.y) + static_cast<double>(b.y),
                        static_cast<double>(a.z) + static_cast<double>(b.z));
  }
  __device__ __forceinline__ void force64(int i, double fx, double fy, double fz,
                                          float scale) const {
    addForce(s, i, static_cast<float>(fx), static_cast<float>(fy), static_cast<float>(fz),
             scale);
  }
  __device__ __forceinline__ void energy64(int k, int slot, double e, float scale) const {
    const long long v = warpSum(__double2ll_rn(e * static_cast<double>(scale)));
    if ((threadIdx.x & 31) == 0 && v != 0) {
      atomicAdd(&s.nrg[k * kNrgStride + slot], static_cast<unsigned long long>(v));
    }
  }
  __device__ __forceinline__ float2 clash(int k) const { return s.clash[k]; }
};

template <bool FORCE, bool ENERGY, class V, bool CLASH = false>
__device__ void valenceTerms(const DevSynthesis &d, const V &v) {
  const float fs = d.frc_scale;
  const float es = d.nrg_scale;
  const int lane = threadIdx.x & 31;
  const int nbond = v.chunks(kBondTerms), nangl = v.chunks(kAnglTerms);
  const int ndihe = v.chunks(kDiheTerms);

  // bonds, valence_potential.tpp:9-97; the equilibrium length is a float pair so that r - r0
  // loses nothing to the rounding of r0, and the bond length itself is an unevaluated pair
  for (int c = v.begin(ndihe + nangl); c < nbond; c += v.chunkStride()) {
    const ValenceTerm t = v.term(kBondTerms, c, lane);
    const int k = t.k;
    float e = 0.0f;
    if (t.valid) {
      const uint4 rec = d.bonds[t.index];
      const int ia = v.slot0(k) + static_cast<int>(rec.x & 0xffffu);
      const int ja = v.slot0(k) + static_cast<int>(rec.x >> 16);
      const float keq = __uint_as_float(rec.y);
      const float leq_hi = __uint_as_float(rec.z);
      const float leq_lo = __uint_as_float(rec.w);
      const float3 ai = v.hi(ia), aj = v.hi(ja), bi = v.lo(ia), bj = v.lo(ja);
      const float av[3] = {aj.x, aj.y, aj.z};
      const float bv[3] = {ai.x, ai.y, ai.z};
      const float lav[3] = {bj.x, bj.y, bj.z};
      const float lbv[3] = {bi.x, bi.y, bi.z};
      float dh[3], dlo[3];
#pragma unroll
      for (int q = 0; q < 3; q++) {
        const float sdiff = av[q] - bv[q];
        const float bb = sdiff - av[q];
        const float err = (av[q] - (sdiff - bb)) + (-bv[q] - bb);
        const float lo = err + (lav[q] - lbv[q]);
        dh[q] = sdiff + lo;
        dlo[q] = lo - (dh[q] - sdiff);
      }
      float r2h = dh[0] * dh[0];
      float r2l = fmaf(dh[0], dh[0], -r2h) + 2.0f * dh[0] * dlo[0];
#pragma unroll
      for (int q = 1; q < 3; q++) {
        const float p = dh[q] * dh[q];
        const float pe = fmaf(dh[q], dh[q], -p) + 2.0f * dh[q] * dlo[q];
        const float sum = r2h + p;
        const float bvv = sum - r2h;
        r2l += ((r2h - (sum - bvv)) + (p - bvv)) + pe;
        r2h = sum;
      }
      const float r = sqrtf(r2h);
      const float r_lo = (fmaf(-r, r, r2h) + r2l) / (2.0f * r);
      const float dl = ((r - leq_hi) + r_lo) - leq_lo;
      if (FORCE) {
        const float fmag = 2.0f * keq * dl / r;
        v.force(ia, fmag * dh[0], fmag * dh[1], fmag * dh[2], fs);
        v.force(ja, -fmag * dh[0], -fmag * dh[1], -fmag * dh[2], fs);
      }
      e = __fmul_rn(__fmul_rn(keq, dl), dl);
    }
    if (ENERGY) {
      v.energy(k, kBond, e, es);
    }
  }

  // angles, valence_potential.tpp:170-288, in FP64 from the exact coordinates: a near-linear
  // angle's force divides by sin(theta), which FP32 deltas and cross products only give to
  // about 1e-7 absolute.  theta - theta0 comes from rotating (cos, sin) of theta, taken from the
  // dot and cross products, by theta0: well conditioned everywhere.
  for (int c = v.begin(ndihe); c < nangl; c += v.chunkStride()) {
    const ValenceTerm t = v.term(kAnglTerms, c, lane);
    const int k = t.k;
    double e = 0.0;
    if (t.valid) {
      const uint4 rec = d.angles[t.index];
      const double4 prm = d.angl64[t.index];   // k, cos, sin, theta0
      const int ia = v.slot0(k) + static_cast<int>(rec.x & 0xffffu);
      const int ja = v.slot0(k) + static_cast<int>(rec.x >> 16);
      const int ka = v.slot0(k) + static_cast<int>(rec.y);
      const double3 pj = v.pos64(ja);
      const double3 ba = sub3d(v.pos64(ia), pj);
      const double3 bc = sub3d(v.pos64(ka), pj);
      // reciprocal square roots instead of divisions and square roots (FP64 divisions are long
      // instruction sequences): 1 / sin(theta) = |ba| |bc| / |ba x bc|
      const double mgba = dot3d(ba, ba);
      const double mgbc = dot3d(bc, bc);
      const double inv_ba = rsqrt(mgba);
      const double inv_bc = rsqrt(mgbc);
      const double invbabc = inv_ba * inv_bc;
      const double3 cr = cross3d(ba, bc);
      const double cr2 = dot3d(cr, cr);
      const double inv_cr = rsqrt(cr2);
      const double sth = cr2 * inv_cr * invbabc;
      const double cth = dot3d(ba, bc) * invbabc;
      const double dtheta = atan2(fma(sth, prm.y, -cth * prm.z), fma(cth, prm.y, sth * prm.z));
      if (FORCE) {
        const double dA = -2.0 * prm.x * dtheta * inv_cr * ((mgba * inv_ba) * (mgbc * inv_bc));
        const double sqba = dA * inv_ba * inv_ba;
        const double sqbc = dA * inv_bc * inv_bc;
        const double mbabc = dA * invbabc;
        const double adx = bc.x * mbabc - cth * ba.x * sqba;
        const double ady = bc.y * mbabc - cth * ba.y * sqba;
        const double adz = bc.z * mbabc - cth * ba.z * sqba;
        const double cdx = ba.x * mbabc - cth * bc.x * sqbc;
        const double cdy = ba.y * mbabc - cth * bc.y * sqbc;
        const double cdz = ba.z * mbabc - cth * bc.z * sqbc;
        v.force64(ia, -adx, -ady, -adz, fs);
        v.force64(ja, adx + cdx, ady + cdy, adz + cdz, fs);
        v.force64(ka, -cdx, -cdy, -cdz, fs);
      }
      e = prm.x * dtheta * dtheta;
    }
    if (ENERGY) {
      v.energy64(k, kAngle, e, es);
    }
  }

  // dihedrals with attached 1-4 pairs, valence_potential.tpp:359-578, 1288-1420, in FP64 from
  // the exact coordinates.  The signed angle is carried as (cos, sin) from x = (ab x bc) .
  // (bc x cd) and y = |bc| ab . (bc x cd), the angle STORMM's acos / arcsine route gives
  // (Math/rounding.tpp:25-80) without its ill conditioning near 0 and pi; cos(n theta - phase)
  // and sin(n theta - phase) follow from the multiple-angle recurrence for integer
  // periodicities.  1 + cos(psi) cancels near psi = pi (impropers, and propers near their
  // minimum); there sin^2(psi) / (1 - cos(psi)) gives the same value without the cancellation.
  for (int c = v.begin(0); c < ndihe; c += v.chunkStride()) {
    const ValenceTerm t = v.term(kDiheTerms, c, lane);
    const int k = t.k;
    double e_prop = 0.0, e_impr = 0.0, e_el14 = 0.0, e_lj14 = 0.0;
    if (t.valid) {
      const uint4 ra = d.dihe_a[t.index];
      const double4 prm = d.dihe64[t.index];     // amplitude, cos(phase), sin(phase), periodicity
      const double4 p14 = d.dihe14_64[t.index];  // the attached 1-4 pair: q q / scee, A, B, flag
      const int li = static_cast<int>(ra.x & 0xffffu);
      const int ll = static_cast<int>((ra.y >> 16) & 0x7fffu);
      const int ia = v.slot0(k) + li;
      const int ja = v.slot0(k) + static_cast<int>(ra.x >> 16);
      const int ka = v.slot0(k) + static_cast<int>(ra.y & 0xffffu);
      const int la = v.slot0(k) + ll;
      const bool improper = (ra.y & 0x80000000u) != 0u;
      const double3 pi = v.pos64(ia);
      const double3 pj = v.pos64(ja);
      const double3 pk = v.pos64(ka);
      const double3 pl = v.pos64(la);
      const double3 ab = sub3d(pj, pi);
      const double3 bc = sub3d(pk, pj);
      const double3 cd = sub3d(pl, pk);
      // attached 1-4 pair between atoms i and l, its attenuated FP64 parameters stored with
      // the term; evaluated first, so that the atoms' positions are no longer live in the
      // torsion's force, and its force joins the torsion's on atoms i and l (one set of
      // accumulator atomics for both)
      double3 f14 = make_double3(0.0, 0.0, 0.0);
      if (p14.w != 0.0) {
        const double3 dv = sub3d(pl, pi);
        const double qiqj = p14.x;
        const double lja = p14.y;
        const double ljb = p14.z;
        const double invr = rsqrt(dot3d(dv, dv));
        const double invr2 = invr * invr;
        const double invr6 = invr2 * invr2 * invr2;
        const float2 cl = CLASH ? v.clash(k) : make_float2(0.0f, 0.0f);
        double fmag = 0.0;
        if (CLASH && (cl.x > 0.0f || cl.y > 0.0f)) {
          // clash-softened 1-4 pair (valence_potential.tpp:1337-1357)
          fmag = softCorePair64(1.0 / invr, invr, qiqj, lja, ljb, cl.x, quadraticCore64(cl.x),
                                cl.y, &e_el14, &e_lj14);
        }
        else {
          if (FORCE) {
            fmag = -(qiqj * invr * invr2) + (6.0 * ljb - 12.0 * lja * invr6) * invr6 * invr2;
          }
          e_el14 = qiqj * invr;
          e_lj14 = (lja * invr6 - ljb) * invr6;
        }
        f14 = make_double3(fmag * dv.x, fmag * dv.y, fmag * dv.z);
      }
      double3 crabbc = cross3d(ab, bc);
      double3 crbccd = cross3d(bc, cd);
      const double bc2 = dot3d(bc, bc);
      const double invbc = rsqrt(bc2);
      const double mgbc = bc2 * invbc;
      const double xx = dot3d(crabbc, crbccd);
      const double yy = mgbc * dot3d(ab, crbccd);
      const double inv_rr = rsqrt(fma(xx, xx, yy * yy));
      const double c1 = xx * inv_rr;
      const double s1 = yy * inv_rr;
      double cn, sn;
      const double freq = prm.w;
      const int nint = static_cast<int>(freq);
      if (static_cast<double>(nint) == freq && nint >= 1 && nint <= 6) {
        cn = c1;
        sn = s1;
        for (int m = 1; m < nint; m++) {
          const double cnew = cn * c1 - sn * s1;
          sn = sn * c1 + cn * s1;
          cn = cnew;
        }
      }
      else {
        sincos(freq * atan2(yy, xx), &sn, &cn);
      }
      const double cos_sangle = cn * prm.y + sn * prm.z;
      const double sin_sangle = sn * prm.y - cn * prm.z;
      const double opc = (cos_sangle >= 0.0) ? 1.0 + cos_sangle :
                                               sin_sangle * sin_sangle / (1.0 - cos_sangle);
      if (improper) {
        e_impr = prm.x * opc;
      }
      else {
        e_prop = prm.x * opc;
      }
      if (FORCE) {
        const double fr = prm.x * freq * sin_sangle;
        const double ab2 = dot3d(ab, ab);
        const double cd2 = dot3d(cd, cd);
        const double invab = rsqrt(ab2);
        const double invcd = rsqrt(cd2);
        const double mgab = ab2 * invab;
        const double cosb = -dot3d(ab, bc) * invab * invbc;
        const double cosc = -dot3d(bc, cd) * invbc * invcd;
        const double isinb2 = (cosb * cosb < kAsymptoticToOne) ?
                              fr * __drcp_rn(1.0 - cosb * cosb) : fr * kInvOneMinusAsymptote;
        const double isinc2 = (cosc * cosc < kAsymptoticToOne) ?
                              fr * __drcp_rn(1.0 - cosc * cosc) : fr * kInvOneMinusAsymptote;
        const double invabc = invab * invbc;
        const double invbcd = invbc * invcd;
        crabbc = make_double3(crabbc.x * invabc, crabbc.y * invabc, crabbc.z * invabc);
        crbccd = make_double3(crbccd.x * invbcd, crbccd.y * invbcd, crbccd.z * invbcd);
        const double fa = -invab * isinb2;
        const double fb1 = (mgbc - mgab * cosb) * invabc * isinb2;
        const double fb2 = cosc * invbc * isinc2;
        const double fd = -invcd * isinc2;
        // each atom's force goes out as soon as it is formed (fewer doubles live at once); the
        // third atom takes minus the sum of the torsion's other three, (fb2 + fd) cd' -
        // (fa + fb1) ab'
        v.force64(ia, crabbc.x * fa + f14.x, crabbc.y * fa + f14.y, crabbc.z * fa + f14.z, fs);
        v.force64(la, -fd * crbccd.x - f14.x, -fd * crbccd.y - f14.y, -fd * crbccd.z - f14.z, fs);
        v.force64(ja, fb1 * crabbc.x - fb2 * crbccd.x, fb1 * crabbc.y - fb2 * crbccd.y,
                  fb1 * crabbc.z - fb2 * crbccd.z, fs);
        const double gab = fa + fb1;
        const double gcd = fb2 + fd;
        v.force64(ka, gcd * crbccd.x - gab * crabbc.x, gcd * crbccd.y - gab * crabbc.y,
                  gcd * crbccd.z - gab * crabbc.z, fs);
      }
    }
    if (ENERGY) {
      v.energy64(k, kProperDihedral, e_prop, es);
      v.energy64(k, kImproperDihedral, e_impr, es);
      v.energy64(k, kElec14, e_el14, es);
      v.energy64(k, kVdw14, e_lj14, es);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Tile walks
// ------------------------------------------------------------------------------------------------
struct TileInfo {
  int k;        // unit molecule
  int ibase;    // first slot of block I
  int jbase;    // first slot of block J
  int ni;       // valid atoms in block I
  int nj;       // valid atoms in block J
  bool diag;
  int local;    // tile index within the molecule
};

__device__ __forceinline__ TileInfo tileInfo(const UnitSmem &s, int nsys_u, int t) {
  TileInfo ti;
  ti.k = findOwner(s.meta + kMetaTile * s.metaStride, nsys_u, t);
  ti.local = t - unitMeta(s, kMetaTile, ti.k);
  int I, J;
  tileCoordinates(ti.local, &I, &J);
  const int n = s.natom[ti.k];
  ti.ibase = s.slot0[ti.k] + I * kTile;
  ti.jbase = s.slot0[ti.k] + J * kTile;
  ti.ni = min(kTile, n - I * kTile);
  ti.nj = min(kTile, n - J * kTile);
  ti.diag = (I == J);
  return ti;
}

// How a warp walks a tile.  Lane l = 16 h + p holds atom il of block I and meets record
// (q + k) mod 16 of block J at step k, that is atoms q and q + 16:
//   off-diagonal                       il = l, q = p, 16 steps: all 32 atoms of block J
//   off-diagonal, at most 16 atoms     il = p, q = p + 8 h, 8 steps: each half warp takes half of
//   in block I                         the records
//   diagonal                           il = l, q = p, 9 steps: a lane's own half of the block at
//                                      distances 1 to 8, the other half at distances 0 to 7 (h = 0)
//                                      or 1 to 8 (h = 1), so that every pair is met once
//   diagonal, at most 16 atoms         il = p, q = p + 1 + 4 h, 4 steps: distances 1 to 4 (h = 0)
//                                      and 5 to 8 (h = 1)
// The traveling accumulators of a record pass from lane to lane within the half warp; after the
// walk, `partner` is the lane of the other half that holds sums of the same record.
struct TileWalk {
  int il;
  int q;
  int steps;
  int partner;
  bool narrow;
  bool diag;
};

__device__ __forceinline__ TileWalk tileWalk(const TileInfo &ti, int lane) {
  const int p = lane & 15, h = lane >> 4;
  TileWalk w;
  w.diag = ti.diag;
  w.narrow = ti.ni <= kRecords;
  const int offset = w.narrow ? (ti.diag ? 1 + 4 * h : 8 * h) : 0;
  const int ahead = w.narrow ? (ti.diag ? (h != 0 ? 4 : -4) : 8) : 0;
  w.il = w.narrow ? p : lane;
  w.q = (p + offset) & 15;
  w.steps = w.narrow ? (ti.diag ? 4 : 8) : (ti.diag ? 9 : 16);
  w.partner = ((h ^ 1) << 4) | ((p + ahead) & 15);
  return w;
}

// Weights (1 or 0) of the two pairs of step k of a diagonal tile
__device__ __forceinline__ float2 diagonalWeights(const TileWalk &w, int lane, int k) {
  const int p = lane & 15, h = lane >> 4;
  if (w.narrow) {
    // atoms q + 16 are padding, which needs no mask
    return f2((k == 3 && h == 1 && p >= 8) ? 0.0f : 1.0f, 1.0f);
  }
  if (k == 0) {
    return f2(0.0f, h == 0 ? 1.0f : 0.0f);
  }
  if (k == 8) {
    return f2((h == 1 || p < 8) ? 1.0f : 0.0f, (h == 1 && p < 8) ? 1.0f : 0.0f);
  }
  return f2(1.0f, 1.0f);
}

// Run one tile: p.pair<false, .>(record, q, 1) for every step, or p.pair<true, .>(record, q,
// weights) where pairs of weight 0 are to be left out, and p.rotate(source lane) after it. Padding
// slots hold parameters that make every contribution to a real atom exactly zero (no charge, zero
// screened radius and dE/dR, masked Lennard-Jones, far-away coordinates), so partial tiles run the
// same branch-free loop.
//
// tileFlush(p) runs after at most eight steps and at the end of the tile: passes that sum energies
// in FP32 move their partial sums into FP64 there, so no FP32 running sum spans more than eight
// pairs of each of the two (the generic overload does nothing).
template <class P>
__device__ __forceinline__ void tileFlush(P &) {}

// PLAIN (off-diagonal tiles of the tiled path): no pair of the tile is masked or closer than the
// distances of tilePlain(), so the passes leave out what only near pairs need.
template <bool PLAIN = false, class P>
__device__ __forceinline__ void walkTile(P &p, const TileInfo &ti, const TileWalk &w, int lane) {
  const int jrec = slotRecord(ti.jbase);
  const int src = (lane & 16) | ((lane + 1) & 15);
  int q = w.q;
  if (PLAIN || !w.diag) {
#pragma unroll 1
    for (int k0 = 0; k0 < w.steps; k0 += 8) {
#pragma unroll P::kUnroll
      for (int k = 0; k < 8; k++) {
        p.template pair<false, PLAIN>(jrec + q, q, f2(1.0f));
        p.rotate(src);
        q = (q + 1) & 15;
      }
      tileFlush(p);
    }
  }
  else {
#pragma unroll 1
    for (int k = 0; k < w.steps; k++) {
      p.template pair<true, false>(jrec + q, q, diagonalWeights(w, lane, k));
      p.rotate(src);
      q = (q + 1) & 15;
      if (k == 4) {
        tileFlush(p);
      }
    }
    tileFlush(p);
  }
}

// Block J's atom whose traveling sum jShare() leaves with this lane after the walk
__device__ __forceinline__ int sharedAtom(const TileWalk &w, int lane) {
  return ((w.q + w.steps) & 15) + (lane & 16);
}

// The two half warps' sums of a record's two atoms: half h takes atom q + 16 h's
__device__ __forceinline__ float jShare(float2 acc, const TileWalk &w, int lane) {
  const bool upper = (lane & 16) != 0;
  const float other = __shfl_sync(kFullMask, upper ? acc.x : acc.y, w.partner);
  return (upper ? acc.y : acc.x) + other;
}

// Block I's atom's sum over a lane's two pairs, and over both half warps where both hold the atom
// (the lanes of the lower half commit it)
__device__ __forceinline__ float iShare(float2 acc, const TileWalk &w) {
  const float v = acc.x + acc.y;
  return w.narrow ? v + __shfl_xor_sync(kFullMask, v, 16) : v;
}

// Whether this lane commits block I's atom il
__device__ __forceinline__ bool ownsAtom(const TileInfo &ti, const TileWalk &w, int lane) {
  return lane < ti.ni && w.il == lane;
}

// Atom i's coordinates, negated and in both halves of a packed pair
struct AtomI {
  float2 hx, hy, hz, lx, ly, lz;
  __device__ __forceinline__ void load(const UnitSmem &s, int slot) {
    const float3 h = slotHi(s, slot), l = slotLo(s, slot);
    hx = f2(-h.x);
    hy = f2(-h.y);
    hz = f2(-h.z);
    lx = f2(-l.x);
    ly = f2(-l.y);
    lz = f2(-l.z);
  }
};

// Separations j - i of a record's two atoms, and their squares' sum; with GUARD, pairs of weight 0
// are put 1e4 A apart
struct Separation2 {
  float2 hx, hy, hz, lx, ly, lz;   // of the hi and lo parts
  float2 dx, dy, dz, r2;
};

template <bool GUARD>
__device__ __forceinline__ Separation2 separate2(const AtomI &i, float4 a, float4 b, float4 c,
                                                 float4 d, float2 w) {
  Separation2 v;
  v.hx = add2(f2(a.x, a.y), i.hx);
  v.hy = add2(f2(a.z, a.w), i.hy);
  v.hz = add2(f2(b.x, b.y), i.hz);
  v.lx = add2(f2(c.x, c.y), i.lx);
  v.ly = add2(f2(c.z, c.w), i.ly);
  v.lz = add2(f2(d.x, d.y), i.lz);
  v.dx = add2(v.hx, v.lx);
  v.dy = add2(v.hy, v.ly);
  v.dz = add2(v.hz, v.lz);
  v.r2 = fma2(v.dx, v.dx, fma2(v.dy, v.dy, mul2(v.dz, v.dz)));
  if (GUARD) {
    v.r2 = f2(w.x != 0.0f ? v.r2.x : 1.0e8f, w.y != 0.0f ? v.r2.y : 1.0e8f);
  }
  return v;
}

// Pairs set aside by a pass, spread over the warp: every lane's bits in `late` (bit k for the
// first pair of step k, bit 16 + k for the second) become entries lane | bit << 5 of the warp's
// list, and f(lane, bit) runs for each, one a lane, so that the few pairs of a tile take one or
// two rounds where lane by lane the busiest lane would set the count.
template <class F>
__device__ __forceinline__ void spreadLate(unsigned late, unsigned short* list, int lane,
                                           const F &f) {
  while (__any_sync(kFullMask, late != 0u)) {
    const int mine = __popc(late);
    int end = mine;                       // inclusive prefix sum over the lanes
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(kFullMask, end, o);
      end += (lane >= o) ? v : 0;
    }
    const int total = min(__shfl_sync(kFullMask, end, 31), kLateEntries);
    for (int at = end - mine; late != 0u && at < kLateEntries; at++) {
      const int b = __ffs(late) - 1;
      late &= late - 1u;
      list[at] = static_cast<unsigned short>(lane | (b << 5));
    }
    __syncwarp();
    for (int e = lane; e < total; e += 32) {
      f(list[e] & 31, list[e] >> 5);
    }
    __syncwarp();
  }
}

// Slots of a pair set aside by lane `of` at bit b, and its step
struct LatePair {
  int islot, jslot, step;
  float2 rho, sj;      // (rho_i, rho_j), (s_j rho_j, s_i rho_i)
  float r, r2, invr;
  float3 dv;           // j - i
  __device__ __forceinline__ LatePair(const UnitSmem &s, const TileInfo &ti, int of, int b) {
    const TileWalk w = tileWalk(ti, of);
    step = b & 15;
    islot = ti.ibase + w.il;
    jslot = ti.jbase + ((w.q + step) & 15) + (b & 16);
    dv = slotDelta(s, islot, jslot);
    r2 = fmaf(dv.x, dv.x, fmaf(dv.y, dv.y, dv.z * dv.z));
    invr = rsqrtf(r2);
    r = r2 * invr;
    rho = f2(slotValue(s.pd, islot, 2), slotValue(s.pd, jslot, 2));
    sj = f2(slotValue(s.pb, jslot, 2), slotValue(s.pb, islot, 2));
  }
};

// GB pass 1: psi_i -= H(r, rho_i, s_j rho_j) and psi_j -= H(r, rho_j, s_i rho_i).  STORE (a force
// evaluation of the fused kernel): the radial derivatives of both terms go to the store for pass 3,
// one float4 per lane and step of the tile walk, so the stores of a step are one coalesced 512-byte
// line.  Pairs that hctSeries2 leaves out are marked in `late` and evaluated by finish() after the
// walk.
template <bool STORE, bool NECK = false, bool BRANCH = false>
struct RadiiPass {
  static constexpr int kUnroll = 2;
  const UnitSmem &s;
  NeckGb neck;
  AtomI at;
  float2 rho_i, s_i;    // radius and screened radius of atom i
  int ni;               // neck index of atom i
  int jneck;            // slot of block J's first atom
  float2 psi_i, psi_j;  // i-side sums, traveling j-side sums
  unsigned late, bit;   // pairs left to finish(), bit of the current step
  float4* out;          // this lane's entry of the store for the current step
  __device__ RadiiPass(const UnitSmem &s_in, const DevSynthesis &d) : s(s_in), neck(d) {}
  __device__ __forceinline__ void begin(const TileInfo &ti, const TileWalk &w,
                                        float4* tile_out = nullptr) {
    const int islot = ti.ibase + w.il;
    at.load(s, islot);
    rho_i = f2(slotValue(s.pd, islot, 2));
    s_i = f2(slotValue(s.pb, islot, 2));
    if (NECK) {
      ni = s.neck[islot];
      jneck = ti.jbase;
    }
    psi_i = f2(0.0f);
    psi_j = f2(0.0f);
    late = 0u;
    bit = 1u;
    out = tile_out;
  }
  template <bool GUARD, bool PLAIN>
  __device__ __forceinline__ void pair(int rec, int q, float2 wt) {
    const float4 a = s.pa[rec], b = s.pb[rec], c = s.pc[rec], d = s.pd[rec];
    const Separation2 v = separate2<GUARD>(at, a, b, c, d, wt);
    const float2 invr = f2(rsqrtf(v.r2.x), rsqrtf(v.r2.y));
    const float2 r = mul2(v.r2, invr);
    const float2 rho_j = f2(d.z, d.w), s_j = f2(b.z, b.w);
    float2 hi, hj, di = f2(0.0f), dj = f2(0.0f);
    const Near2 late_i = hctSeries2<STORE, BRANCH, PLAIN>(r, invr, rho_i, s_j, &hi, &di);
    const Near2 late_j = hctSeries2<STORE, BRANCH, PLAIN>(r, invr, rho_j, s_i, &hj, &dj);
    const bool late_x = late_i.x || late_j.x;
    const bool late_y = late_i.y || late_j.y;
    if (NECK && !PLAIN) {
      if (!late_x && r.x < rho_i.x + rho_j.x + neck.reach) {
        const int nj = s.neck[jneck + q];
        float e, f;
        hi.x += neck.both(ni, nj, r.x, invr.x, &e);
        hj.x += neck.both(nj, ni, r.x, invr.x, &f);
        di.x += e;
        dj.x += f;
      }
      if (!late_y && r.y < rho_i.y + rho_j.y + neck.reach) {
        const int nj = s.neck[jneck + q + 16];
        float e, f;
        hi.y += neck.both(ni, nj, r.y, invr.y, &e);
        hj.y += neck.both(nj, ni, r.y, invr.y, &f);
        di.y += e;
        dj.y += f;
      }
    }
    late |= (late_x ? bit : 0u) | (late_y ? bit << 16 : 0u);
    // a select, not a weight of zero: the series grows as r^-20 and overflows where two atoms
    // nearly coincide (below 0.015 A for a screened radius of 1.4), and zero times that is NaN
    const float2 neg = GUARD ? f2(-wt.x, -wt.y) : f2(-1.0f);
    psi_i = fma2(f2(late_x ? 0.0f : hi.x, late_y ? 0.0f : hi.y), neg, psi_i);
    psi_j = fma2(f2(late_x ? 0.0f : hj.x, late_y ? 0.0f : hj.y), neg, psi_j);
    if (STORE) {
      __stcg(out, make_float4(di.x, di.y, dj.x, dj.y));
    }
  }
  __device__ __forceinline__ void rotate(int src) {
    psi_j.x = __shfl_sync(kFullMask, psi_j.x, src);
    psi_j.y = __shfl_sync(kFullMask, psi_j.y, src);
    bit <<= 1;
    if (STORE) {
      out += 32;
    }
  }
  // The pairs left out, after the walk; add(slot, v) adds v to a slot's descreening sum, and
  // tile_out is the tile's first entry of the store
  template <class Add>
  __device__ __forceinline__ void finish(const TileInfo &ti, int lane, unsigned short* list,
                                         float4* tile_out, const Add &add) const {
    spreadLate(late, list, lane, [&](int of, int b) {
      const LatePair p(s, ti, of, b);
      const float4 c = hctClosed2<STORE>(p.r, p.r2, p.invr, p.rho, p.sj);
      float2 h = f2(c.x, c.y), hd = f2(c.z, c.w);
      if (NECK && p.r < p.rho.x + p.rho.y + neck.reach) {
        const int a = s.neck[p.islot], z = s.neck[p.jslot];
        float e, f;
        h.x += neck.both(a, z, p.r, p.invr, &e);
        h.y += neck.both(z, a, p.r, p.invr, &f);
        hd.x += e;
        hd.y += f;
      }
      add(p.islot, -h.x);
      add(p.jslot, -h.y);
      if (STORE) {
        float* entry = reinterpret_cast<float*>(tile_out + 32 * p.step + of) + (b >> 4);
        __stcg(entry, hd.x);
        __stcg(entry + 2, hd.y);
      }
    });
  }
};

// Pass 2: Coulomb + Lennard-Jones on non-excluded pairs and the GB pair terms; with CLASH, the
// Coulomb and Lennard-Jones terms of a molecule given a clash distance or ratio take softened
// cores (the uniform branch is per tile: a tile belongs to one molecule).  Energies are summed
// negated (flush turns them), and both sides' forces as fmag x (r_j - r_i): block I's as they are,
// block J's to be negated by the caller.
template <bool FORCE, bool ENERGY, bool NB, bool GB, bool CLASH = false>
struct PairPass {
  static constexpr int kUnroll = 2;
  const UnitSmem &s;
  float kk, inv_diel;
  bool salt;
  AtomI at;
  float2 q_i, r_i;  // charge and effective radius of atom i
  float2 m4r_i;     // -1 / (4 R_i)
  int code_i;
  unsigned mask;
  bool soft;        // softened cores on this tile
  float clash_d, clash_r;
  float2 qcore;
  float2 fxi, fyi, fzi, dei, fxj, fyj, fzj, dej;
  float2 e_elec, e_vdw, e_gb;       // FP32 sums of at most eight pairs each (see tileFlush)
  double t_elec, t_vdw, t_gb;       // this lane's FP64 sums over the tile (see tileEnergy)
  __device__ PairPass(const UnitSmem &s_in, float kappa, float inv_dielectric) :
      s(s_in), kk(-kappa * kGbKscale), inv_diel(inv_dielectric), salt(kappa > 0.0f) {}
  __device__ __forceinline__ void flush() {
    if (ENERGY) {
      if (NB) {
        t_elec -= static_cast<double>(e_elec.x) + static_cast<double>(e_elec.y);
        t_vdw -= static_cast<double>(e_vdw.x) + static_cast<double>(e_vdw.y);
      }
      if (GB) {
        t_gb -= static_cast<double>(e_gb.x) + static_cast<double>(e_gb.y);
      }
      e_elec = e_vdw = e_gb = f2(0.0f);
    }
  }
  __device__ __forceinline__ void begin(const TileInfo &ti, const TileWalk &w, unsigned mask_in,
                                        float2 clash = make_float2(0.0f, 0.0f)) {
    const int islot = ti.ibase + w.il;
    at.load(s, islot);
    q_i = f2(slotValue(s.pb, islot, 2));
    r_i = f2(slotValue(s.pd, islot, 2));
    m4r_i = f2(-0.25f * slotValue(s.pg, islot, 0));
    code_i = __float_as_int(slotValue(s.pg, islot, 2)) & 0xffff;
    mask = mask_in;
    if (CLASH) {
      clash_d = clash.x;
      clash_r = clash.y;
      soft = (clash.x > 0.0f || clash.y > 0.0f);
      qcore = quadraticCore(clash.x);
    }
    fxi = fyi = fzi = dei = f2(0.0f);
    fxj = fyj = fzj = dej = f2(0.0f);
    e_elec = e_vdw = e_gb = f2(0.0f);
    t_elec = t_vdw = t_gb = 0.0;
  }
  template <bool GUARD, bool PLAIN>
  __device__ __forceinline__ void pair(int rec, int q, float2 wt) {
    const float4 a = s.pa[rec], b = s.pb[rec], c = s.pc[rec], d = s.pd[rec], g = s.pg[rec];
    const Separation2 v = separate2<GUARD>(at, a, b, c, d, wt);
    const float2 r2 = v.r2;
    float2 qq = mul2(q_i, f2(b.z, b.w));
    if (GUARD) {
      qq = mul2(qq, wt);
    }
    float2 fmag = f2(0.0f);
    if (NB) {
      // excluded and padding pairs take the same path with zero parameters; nincl is -1 or 0
      const unsigned m = mask >> q;
      float2 nincl = PLAIN ? f2(-1.0f) :
                             f2((m & 1u) ? 0.0f : -1.0f, (m & 0x10000u) ? 0.0f : -1.0f);
      if (GUARD) {
        nincl = mul2(nincl, wt);
      }
      // 1/r from rsqrt with one Newton step (Coulomb), and 1/r^2 as its own reciprocal: r^-6
      // and r^-12 multiply the relative error of 1/r^2 by 3 and 6, so squaring 1/r (twice its
      // error) would double the rounding of the repulsive wall, and the Newton step of 1/r^2
      // takes the exact r^2 = r2 + 2 (dx ex + dy ey + dz ez) + O(e^2), the e the separations'
      // recovered rounding errors (splitCoordinate): without it the Lennard-Jones energy of a
      // molecule with close contacts errs by up to 1.5e-6 of the root-sum-square of its pair
      // terms.  r2 >= 256 on padding slots, never zero.  Beyond the distance of a plain tile the
      // Lennard-Jones term is below 1e-5 of a contact's and takes the square of 1/r: over 30 chains
      // of 2,500 atoms and four batches of 32 chains the errors against the FP64 mode are the same
      // to three digits either way (forces of the pair terms 2.5e-7 and 2.8e-7, Lennard-Jones
      // energy 7.8e-8 and 6.0e-8), and 32 chains take 1,304 us instead of 1,359.
      float2 invr = f2(rsqrtf(r2.x), rsqrtf(r2.y));
      invr = mul2(invr, fma2(mul2(mul2(r2, f2(-0.5f)), invr), invr, f2(1.5f)));
      float2 invr2;
      if (PLAIN) {
        invr2 = mul2(invr, invr);
      }
      else {
        const float2 ex = sub2(v.lx, sub2(v.dx, v.hx));
        const float2 ey = sub2(v.ly, sub2(v.dy, v.hy));
        const float2 ez = sub2(v.lz, sub2(v.dz, v.hz));
        float2 m2r2c = fma2(v.dx, ex, fma2(v.dy, ey, mul2(v.dz, ez)));
        m2r2c = mul2(m2r2c, f2(-2.0f));
        invr2 = f2(__fdividef(1.0f, r2.x), __fdividef(1.0f, r2.y));
        const float2 step = fma2(m2r2c, invr2, fma2(mul2(r2, f2(-1.0f)), invr2, f2(1.0f)));
        invr2 = fma2(invr2, step, invr2);
      }
      const float2 invr6 = mul2(mul2(invr2, invr2), invr2);
      const float2 ab1 = s.lj[code_i + (__float_as_int(g.z) >> 16)];
      const float2 ab2 = s.lj[code_i + (__float_as_int(g.w) >> 16)];
      const float2 nqq = mul2(qq, nincl);
      const float2 nla = mul2(f2(ab1.x, ab2.x), nincl);
      const float2 nlb = mul2(f2(ab1.y, ab2.y), nincl);
      if (CLASH && soft) {
        float ee = 0.0f, ev = 0.0f;
        fmag.x = softCorePair(r2.x * invr.x, invr.x, -nqq.x, -nla.x, -nlb.x, clash_d, qcore,
                              clash_r, &ee, &ev);
        e_elec.x -= ee;
        e_vdw.x -= ev;
        ee = ev = 0.0f;
        fmag.y = softCorePair(r2.y * invr.y, invr.y, -nqq.y, -nla.y, -nlb.y, clash_d, qcore,
                              clash_r, &ee, &ev);
        e_elec.y -= ee;
        e_vdw.y -= ev;
      }
      else {
        // -(A / r^6 - B)
        const float2 nw = fma2(nla, invr6, mul2(nlb, f2(-1.0f)));
        if (ENERGY) {
          e_elec = fma2(nqq, invr, e_elec);                       // minus the energy
          e_vdw = fma2(nw, invr6, e_vdw);
        }
        if (FORCE) {
          // -(qq / r^3) + (6 B - 12 A / r^6) / r^8
          fmag = mul2(invr2, fma2(nqq, invr, mul2(mul2(invr6, f2(6.0f)), fma2(nla, invr6, nw))));
        }
      }
    }
    if (GB) {
      const float2 ijb = mul2(r_i, f2(d.z, d.w));
      const float2 arg = mul2(mul2(r2, m4r_i), f2(g.x, g.y));
      const float2 efac = f2(__expf(arg.x), __expf(arg.y));
      const float2 f2gb = fma2(ijb, efac, r2);
      const float2 fgbi = f2(rsqrtf(f2gb.x), rsqrtf(f2gb.y));
      float2 dielfac, chain;       // 1 - exp(...) / diel, and the same plus its r derivative's part
      if (salt) {
        const float2 fgbk = f2(__fdividef(kk, fgbi.x), __fdividef(kk, fgbi.y));
        const float2 expmkf = f2(__expf(fgbk.x) * inv_diel, __expf(fgbk.y) * inv_diel);
        dielfac = f2(1.0f - expmkf.x, 1.0f - expmkf.y);
        chain = fma2(fgbk, expmkf, dielfac);
      }
      else {
        dielfac = f2(1.0f - inv_diel);
        chain = dielfac;
      }
      const float2 qf = mul2(qq, fgbi);
      if (ENERGY) {
        e_gb = fma2(qf, dielfac, e_gb);                           // minus the energy
      }
      if (FORCE) {
        const float2 temp6 = mul2(mul2(qf, mul2(fgbi, fgbi)), chain);
        fmag = fma2(temp6, fma2(f2(-0.25f), efac, f2(1.0f)), fmag);
        const float2 temp5 = mul2(mul2(mul2(efac, f2(0.5f)), temp6), fma2(f2(0.25f), r2, ijb));
        dei = fma2(r_i, temp5, dei);
        dej = fma2(f2(d.z, d.w), temp5, dej);
      }
    }
    if (FORCE) {
      fxi = fma2(fmag, v.dx, fxi);
      fyi = fma2(fmag, v.dy, fyi);
      fzi = fma2(fmag, v.dz, fzi);
      fxj = fma2(fmag, v.dx, fxj);
      fyj = fma2(fmag, v.dy, fyj);
      fzj = fma2(fmag, v.dz, fzj);
    }
  }
  __device__ __forceinline__ void rotate(int src) {
    if (FORCE) {
      fxj.x = __shfl_sync(kFullMask, fxj.x, src);
      fxj.y = __shfl_sync(kFullMask, fxj.y, src);
      fyj.x = __shfl_sync(kFullMask, fyj.x, src);
      fyj.y = __shfl_sync(kFullMask, fyj.y, src);
      fzj.x = __shfl_sync(kFullMask, fzj.x, src);
      fzj.y = __shfl_sync(kFullMask, fzj.y, src);
      if (GB) {
        dej.x = __shfl_sync(kFullMask, dej.x, src);
        dej.y = __shfl_sync(kFullMask, dej.y, src);
      }
    }
  }
};

template <bool FORCE, bool ENERGY, bool NB, bool GB, bool CLASH>
__device__ __forceinline__ void tileFlush(PairPass<FORCE, ENERGY, NB, GB, CLASH> &p) {
  p.flush();
}

// Pass 3 of the tiled path: radius chain-rule forces, the HCT derivatives evaluated again (the
// pair-derivative store would cost more bytes there than the arithmetic it saves)
template <bool NECK = false>
struct DerivPass {
  static constexpr int kUnroll = 2;
  const UnitSmem &s;
  NeckGb neck;
  AtomI at;
  float2 rho_i, s_i, de_i;
  int ni, jneck;
  unsigned late, bit;
  float2 fxi, fyi, fzi, fxj, fyj, fzj;
  __device__ DerivPass(const UnitSmem &s_in, const DevSynthesis &d) : s(s_in), neck(d) {}
  __device__ __forceinline__ void begin(const TileInfo &ti, const TileWalk &w) {
    const int islot = ti.ibase + w.il;
    at.load(s, islot);
    rho_i = f2(slotValue(s.pd, islot, 2));
    s_i = f2(slotValue(s.pb, islot, 2));
    de_i = f2(slotValue(s.pg, islot, 2));
    if (NECK) {
      ni = s.neck[islot];
      jneck = ti.jbase;
    }
    late = 0u;
    bit = 1u;
    fxi = fyi = fzi = f2(0.0f);
    fxj = fyj = fzj = f2(0.0f);
  }
  __device__ __forceinline__ float neckForce(int a, int z, float r, float invr, float de_a,
                                             float de_z) const {
    float da, dz;
    neck.both(a, z, r, invr, &da);
    neck.both(z, a, r, invr, &dz);
    return da * de_a + dz * de_z;
  }
  template <bool GUARD, bool PLAIN>
  __device__ __forceinline__ void pair(int rec, int q, float2 wt) {
    const float4 a = s.pa[rec], b = s.pb[rec], c = s.pc[rec], d = s.pd[rec], g = s.pg[rec];
    const Separation2 v = separate2<GUARD>(at, a, b, c, d, wt);
    const float2 invr = f2(rsqrtf(v.r2.x), rsqrtf(v.r2.y));
    const float2 r = mul2(v.r2, invr);
    const float2 rho_j = f2(d.z, d.w), s_j = f2(b.z, b.w), de_j = f2(g.z, g.w);
    float2 unused, di, dj;
    const Near2 late_i = hctSeries2<true, true, PLAIN>(r, invr, rho_i, s_j, &unused, &di);
    const Near2 late_j = hctSeries2<true, true, PLAIN>(r, invr, rho_j, s_i, &unused, &dj);
    const bool late_x = late_i.x || late_j.x;
    const bool late_y = late_i.y || late_j.y;
    float2 fmag = fma2(di, de_i, mul2(dj, de_j));
    if (NECK && !PLAIN) {
      if (!late_x && r.x < rho_i.x + rho_j.x + neck.reach) {
        fmag.x += neckForce(ni, s.neck[jneck + q], r.x, invr.x, de_i.x, de_j.x);
      }
      if (!late_y && r.y < rho_i.y + rho_j.y + neck.reach) {
        fmag.y += neckForce(ni, s.neck[jneck + q + 16], r.y, invr.y, de_i.y, de_j.y);
      }
    }
    late |= (late_x ? bit : 0u) | (late_y ? bit << 16 : 0u);
    if (GUARD) {
      fmag = mul2(fmag, wt);
    }
    fmag = f2(late_x ? 0.0f : fmag.x, late_y ? 0.0f : fmag.y);
    fxi = fma2(fmag, v.dx, fxi);
    fyi = fma2(fmag, v.dy, fyi);
    fzi = fma2(fmag, v.dz, fzi);
    fxj = fma2(fmag, v.dx, fxj);
    fyj = fma2(fmag, v.dy, fyj);
    fzj = fma2(fmag, v.dz, fzj);
  }
  __device__ __forceinline__ void rotate(int src) {
    fxj.x = __shfl_sync(kFullMask, fxj.x, src);
    fxj.y = __shfl_sync(kFullMask, fxj.y, src);
    fyj.x = __shfl_sync(kFullMask, fyj.x, src);
    fyj.y = __shfl_sync(kFullMask, fyj.y, src);
    fzj.x = __shfl_sync(kFullMask, fzj.x, src);
    fzj.y = __shfl_sync(kFullMask, fzj.y, src);
    bit <<= 1;
  }
  // The pairs hctSeries2 left out, after the walk; add(slot, fx, fy, fz) adds to a slot's force
  template <class Add>
  __device__ __forceinline__ void finish(const TileInfo &ti, int lane, unsigned short* list,
                                         const Add &add) const {
    spreadLate(late, list, lane, [&](int of, int b) {
      const LatePair p(s, ti, of, b);
      const float4 c = hctClosed2<true>(p.r, p.r2, p.invr, p.rho, p.sj);
      const float de_a = slotValue(s.pg, p.islot, 2), de_z = slotValue(s.pg, p.jslot, 2);
      float fmag = fmaf(c.z, de_a, c.w * de_z);
      if (NECK && p.r < p.rho.x + p.rho.y + neck.reach) {
        fmag += neckForce(s.neck[p.islot], s.neck[p.jslot], p.r, p.invr, de_a, de_z);
      }
      add(p.islot, -fmag * p.dv.x, -fmag * p.dv.y, -fmag * p.dv.z);
      add(p.jslot, fmag * p.dv.x, fmag * p.dv.y, fmag * p.dv.z);
    });
  }
};

// Pass 3 from the stored derivatives: the force of a pair is (hd_i dE/dR_i + hd_j dE/dR_j) times
// the separation, with no transcendental left to evaluate.  Both sides sum +force x separation;
// the caller negates block I's.
struct DerivStoredPass {
  static constexpr int kUnroll = 4;
  const UnitSmem &s;
  AtomI at;
  float2 de_i;
  float2 fxi, fyi, fzi, fxj, fyj, fzj;
  const float4* in;
  __device__ DerivStoredPass(const UnitSmem &s_in) : s(s_in) {}
  __device__ __forceinline__ void begin(const TileInfo &ti, const TileWalk &w,
                                        const float4* tile_in) {
    const int islot = ti.ibase + w.il;
    at.load(s, islot);
    de_i = f2(slotValue(s.pg, islot, 2));
    fxi = fyi = fzi = f2(0.0f);
    fxj = fyj = fzj = f2(0.0f);
    in = tile_in;
  }
  template <bool GUARD, bool PLAIN>
  __device__ __forceinline__ void pair(int rec, int, float2 wt) {
    const float4 hd = __ldcs(in);
    const float4 a = s.pa[rec], b = s.pb[rec], c = s.pc[rec], d = s.pd[rec], g = s.pg[rec];
    const Separation2 v = separate2<false>(at, a, b, c, d, wt);
    float2 fmag = fma2(f2(hd.x, hd.y), de_i, mul2(f2(hd.z, hd.w), f2(g.z, g.w)));
    if (GUARD) {
      fmag = f2(wt.x != 0.0f ? fmag.x : 0.0f, wt.y != 0.0f ? fmag.y : 0.0f);
    }
    fxi = fma2(fmag, v.dx, fxi);
    fyi = fma2(fmag, v.dy, fyi);
    fzi = fma2(fmag, v.dz, fzi);
    fxj = fma2(fmag, v.dx, fxj);
    fyj = fma2(fmag, v.dy, fyj);
    fzj = fma2(fmag, v.dz, fzj);
  }
  __device__ __forceinline__ void rotate(int src) {
    fxj.x = __shfl_sync(kFullMask, fxj.x, src);
    fxj.y = __shfl_sync(kFullMask, fxj.y, src);
    fyj.x = __shfl_sync(kFullMask, fyj.x, src);
    fyj.y = __shfl_sync(kFullMask, fyj.y, src);
    fzj.x = __shfl_sync(kFullMask, fzj.x, src);
    fzj.y = __shfl_sync(kFullMask, fzj.y, src);
    in += 32;
  }
};

// This lane's entry for step 0 of tile t of a unit whose tiles start at tile_base in the store
__device__ __forceinline__ float4* pairDerivTile(const DevSynthesis &d, int tile_base, int t,
                                                 int lane) {
  return d.pair_deriv + static_cast<size_t>(tile_base + t) * kPairDerivPerTile + lane;
}

template <bool STORE, bool NECK>
__device__ void gbRadiiTiles(const DevSynthesis &d, const UnitSmem &s, int nsys_u, int ntiles,
                             int tile_base, int first, int stride) {
  const int lane = threadIdx.x & 31;
  const float ps = static_cast<float>(1 << kPsiBits);
  unsigned short* list = s.late + (threadIdx.x >> 5) * kLateEntries;
  const auto add = [&](int slot, float v) {
    atomicAddInt63(v * ps, &s.psi[slot], &s.psio[slot]);
  };
  RadiiPass<STORE, NECK> p(s, d);
  for (int t = first; t < ntiles; t += stride) {
    const TileInfo ti = tileInfo(s, nsys_u, t);
    const TileWalk w = tileWalk(ti, lane);
    float4* out = STORE ? pairDerivTile(d, tile_base, t, lane) : nullptr;
    p.begin(ti, w, out);
    walkTile(p, ti, w, lane);
    const float vi = iShare(p.psi_i, w);
    const float vj = jShare(p.psi_j, w, lane);
    if (ownsAtom(ti, w, lane)) {
      add(ti.ibase + lane, vi);
    }
    const int jl = sharedAtom(w, lane);
    if (jl < ti.nj) {
      add(ti.jbase + jl, vj);
    }
    p.finish(ti, lane, list, STORE ? out - lane : nullptr, add);
  }
}

template <bool FORCE, bool ENERGY, bool NB, bool GB, bool CLASH = false>
__device__ void pairTiles(const DevSynthesis &d, const UnitSmem &s, int nsys_u, int ntiles,
                          int first, int stride) {
  const int lane = threadIdx.x & 31;
  const float fs = d.frc_scale;
  const float es = d.nrg_scale;
  const float ds = static_cast<float>(1 << kDeijdaBits);
  PairPass<FORCE, ENERGY, NB, GB, CLASH> p(s, d.kappa, d.inv_dielectric);
  // a molecule's energies over this warp's tiles, each tile rounded to the output grid
  // (tileEnergy), the same value in every lane
  long long acc_elec = 0, acc_vdw = 0, acc_gb = 0;
  int acc_k = -1;
  auto commit = [&]() {
    if (lane == 0 && acc_k >= 0) {
      if (NB) {
        atomicAdd(&s.nrg[acc_k * kNrgStride + kElec], static_cast<unsigned long long>(acc_elec));
        atomicAdd(&s.nrg[acc_k * kNrgStride + kVdw], static_cast<unsigned long long>(acc_vdw));
      }
      if (GB) {
        atomicAdd(&s.nrg[acc_k * kNrgStride + kGb], static_cast<unsigned long long>(acc_gb));
      }
    }
    acc_elec = acc_vdw = acc_gb = 0;
  };
  for (int t = first; t < ntiles; t += stride) {
    const TileInfo ti = tileInfo(s, nsys_u, t);
    const TileWalk w = tileWalk(ti, lane);
    if (ENERGY && ti.k != acc_k) {
      commit();
      acc_k = ti.k;
    }
    unsigned mask = 0u;
    if (NB) {
      const int midx = d.tile_mask_idx[unitMeta(s, kMetaMask0, ti.k) + ti.local];
      if (midx != 0) {
        mask = __ldg(&d.mask_pool[static_cast<size_t>(midx) * 32 + w.il]);
      }
    }
    p.begin(ti, w, mask, CLASH ? s.clash[ti.k] : make_float2(0.0f, 0.0f));
    walkTile(p, ti, w, lane);
    if (FORCE) {
      const float fxi = iShare(p.fxi, w), fyi = iShare(p.fyi, w), fzi = iShare(p.fzi, w);
      const float dei = GB ? iShare(p.dei, w) : 0.0f;
      const float fxj = jShare(p.fxj, w, lane), fyj = jShare(p.fyj, w, lane);
      const float fzj = jShare(p.fzj, w, lane);
      const float dej = GB ? jShare(p.dej, w, lane) : 0.0f;
      if (ownsAtom(ti, w, lane)) {
        const int is = ti.ibase + lane;
        addForce(s, is, fxi, fyi, fzi, fs);
        if (GB) {
          atomicAddInt63(dei * ds, &s.de[is], &s.deo[is]);
        }
      }
      const int jl = sharedAtom(w, lane);
      if (jl < ti.nj) {
        const int js = ti.jbase + jl;
        addForce(s, js, -fxj, -fyj, -fzj, fs);
        if (GB) {
          atomicAddInt63(dej * ds, &s.de[js], &s.deo[js]);
        }
      }
    }
    if (ENERGY) {
      if (NB) {
        acc_elec += tileEnergy(p.t_elec, es);
        acc_vdw += tileEnergy(p.t_vdw, es);
      }
      if (GB) {
        acc_gb += tileEnergy(p.t_gb, es);
      }
    }
  }
  if (ENERGY) {
    commit();
  }
}

__device__ void gbDerivativeTiles(const DevSynthesis &d, const UnitSmem &s, int nsys_u,
                                  int ntiles, int tile_base, int first, int stride) {
  const int lane = threadIdx.x & 31;
  const float fs = d.frc_scale;
  DerivStoredPass p(s);
  for (int t = first; t < ntiles; t += stride) {
    const TileInfo ti = tileInfo(s, nsys_u, t);
    const TileWalk w = tileWalk(ti, lane);
    p.begin(ti, w, pairDerivTile(d, tile_base, t, lane));
    walkTile(p, ti, w, lane);
    const float fxi = iShare(p.fxi, w), fyi = iShare(p.fyi, w), fzi = iShare(p.fzi, w);
    const float fxj = jShare(p.fxj, w, lane), fyj = jShare(p.fyj, w, lane);
    const float fzj = jShare(p.fzj, w, lane);
    if (ownsAtom(ti, w, lane)) {
      addForce(s, ti.ibase + lane, -fxi, -fyi, -fzi, fs);
    }
    const int jl = sharedAtom(w, lane);
    if (jl < ti.nj) {
      addForce(s, ti.jbase + jl, fxj, fyj, fzj, fs);
    }
  }
}
// ------------------------------------------------------------------------------------------------
// Per-atom GB steps between the pair passes (nonbonded_potential.tpp:730-805, 982-1021)
// ------------------------------------------------------------------------------------------------
// Effective radius of atom gi from its descreening sum psi (HCT, or OBC / OBC-II)
// Effective GB radius of an atom from its descreening sum psi, in FP64 with the FP64
// parameters: the OBC form 1 / (1 / rho - tanh(...) / r) cancels for buried atoms, where tanh
// nears 1 and 1 / rho - 1 / r is a small difference, and FP32 there loses the 1e-6 relative
// accuracy of the GB energy on compact proteins.  One evaluation per atom, so FP64 costs
// nothing measurable.
__device__ __forceinline__ float effectiveRadius(const DevSynthesis &d, int gi, double psi) {
  const double4 p = d.gb_radius64[gi];   // rho, intrinsic radius, alpha, beta
  double egbi;
  if (d.igb == 1) {
    egbi = 1.0 / (1.0 / p.x + psi);
    if (egbi < 0.0) egbi = 30.0;
  }
  else {
    const double fipsi = psi * (-p.x);
    egbi = 1.0 / (1.0 / p.x - tanh((p.z - p.w * fipsi + d.gb_gamma64[gi] * fipsi * fipsi) *
                                   fipsi) / p.y);
  }
  return static_cast<float>(egbi);
}

// GB self energy of a charge q (scaled by sqrt of the Coulomb constant) with effective radius
// egbi; *self_de receives its dE/dR contribution
__device__ __forceinline__ float gbSelfTerm(const DevSynthesis &d, float q, float egbi,
                                            float* self_de) {
  const float expmkf = ((d.kappa > 0.0f) ? expf(-kGbKscale * d.kappa * egbi) : 1.0f) *
                       d.inv_dielectric;
  const float dielfac = 1.0f - expmkf;
  const float atmq2h = 0.5f * q * q;
  const float atmqd2h = atmq2h * dielfac;
  *self_de = atmqd2h - kGbKscale * d.kappa * atmq2h * expmkf * egbi;
  return -__fdiv_rn(atmqd2h, egbi);
}

// OBC chain-rule factor dR/dpsi-type prefactor applied to the summed dE/dR
// OBC chain-rule factor (the dR/dpsi-type prefactor applied to the summed dE/dR), in FP64 for
// the same reason: 1 - tanh^2 cancels where tanh nears 1
__device__ __forceinline__ float obcChainFactor(const DevSynthesis &d, int gi, double psi) {
  const double4 p = d.gb_radius64[gi];
  const double fipsi = psi * (-p.x);
  const double ga = d.gb_gamma64[gi];
  const double thi = tanh((p.z - (p.w - ga * fipsi) * fipsi) * fipsi);
  return static_cast<float>((p.z - (2.0 * p.w - 3.0 * ga * fipsi) * fipsi) * (1.0 - thi * thi) *
                            p.x / p.y);
}

// ------------------------------------------------------------------------------------------------
// Work-unit staging and the staged evaluation, shared by the evaluation and minimization kernels
// ------------------------------------------------------------------------------------------------
struct UnitShape {
  int nsys;       // molecules in the unit
  int nslots;     // atom slots (sum of the molecules' sizes padded to 32)
  int ntiles;     // 32 x 32 tiles of the molecules' lower triangles
  int tile_base;  // first tile of the unit in the pair-derivative store
};

// Molecule table, prefix sums and Lennard-Jones tables of unit u.  Returns false (after setting
// bit 0 of the status word) when the unit does not fit the launch's shared-memory carve-out; the
// caller then skips the unit.  Ends with a barrier.
template <class Team>
__device__ bool stageUnitTables(const DevSynthesis &d, const UnitSmem &s, int u, int max_lj,
                                UnitShape* shape, const Team &team) {
  const int max_sys = s.metaStride - 1;
  const int4 desc = d.unit_desc[u];
  const int nsys_u = desc.y;
  shape->nsys = nsys_u;
  shape->nslots = desc.z;
  shape->ntiles = desc.w;
  if (nsys_u > max_sys) {
    if (team.rank() == 0) {
      atomicOr(d.status, 1);
    }
    return false;
  }
  // the unit's molecule table, precomputed on the host
  const int* meta = d.unit_meta + static_cast<size_t>(desc.x) * kUnitMetaFields;
  shape->tile_base = meta[nsys_u * kUnitMetaFields + kMetaSystem];
  for (int e = team.rank(); e < (nsys_u + 1) * kUnitMetaFields; e += team.size()) {
    s.meta[(e % kUnitMetaFields) * s.metaStride + e / kUnitMetaFields] = meta[e];
  }
  team.sync();
  const int nlj = unitMeta(s, kMetaLj, nsys_u);
  if (desc.z > d.max_unit_slots || nlj > max_lj || nsys_u > max_sys) {
    if (team.rank() == 0) {
      atomicOr(d.status, 1);
    }
    return false;   // reported through the status word; nothing in the unit is touched
  }
  // Lennard-Jones tables of every molecule, all entries in parallel
  for (int e = team.rank(); e < nlj; e += team.size()) {
    const int k = findOwner(s.meta + kMetaLj * s.metaStride, nsys_u, e);
    s.lj[e] = d.ljab[unitMeta(s, kMetaLjTable, k) + e - unitMeta(s, kMetaLj, k)];
  }
  team.sync();
  return true;
}

// Static per-slot parameters of an atom (a < natom) or of a padding slot: charge, Lennard-Jones
// code, rho, s * rho.  A padding slot has no charge, zero screened radius and a masked
// Lennard-Jones row, so every pair term it enters is exactly zero for the real atom.
__device__ __forceinline__ float4 slotParameters(const DevSynthesis &d, const UnitSmem &s, int k,
                                                 int a) {
  if (a < s.natom[k]) {
    const int gi = unitMeta(s, kMetaAtom0, k) + a;
    const int nt = unitMeta(s, kMetaTypes, k) & 0xff;
    const int ty = d.lj_idx[gi];
    return make_float4(d.charge[gi],
                       __int_as_float((unitMeta(s, kMetaLj, k) + ty * nt) | (ty << 16)),
                       d.rho[gi], d.srho[gi]);
  }
  return make_float4(0.0f, __int_as_float(unitMeta(s, kMetaLj, k)), 1.0f, 0.0f);
}

// Neck GB table index of slot a of unit molecule k (0 for padding or other GB models)
__device__ __forceinline__ int slotNeck(const DevSynthesis &d, const UnitSmem &s, int k, int a) {
  return (d.neck_size > 0 && a < s.natom[k]) ? d.neck_idx[unitMeta(s, kMetaAtom0, k) + a] : 0;
}

// Write a slot's coordinates, payloads and GB values
__device__ __forceinline__ void putSlot(const UnitSmem &s, int slot, float3 hi, float3 lo, float w1,
                                        float w2, float g, float h) {
  slotValue(s.pa, slot, 0) = hi.x;
  slotValue(s.pa, slot, 2) = hi.y;
  slotValue(s.pb, slot, 0) = hi.z;
  slotValue(s.pb, slot, 2) = w1;
  slotValue(s.pc, slot, 0) = lo.x;
  slotValue(s.pc, slot, 2) = lo.y;
  slotValue(s.pd, slot, 0) = lo.z;
  slotValue(s.pd, slot, 2) = w2;
  slotValue(s.pg, slot, 0) = g;
  slotValue(s.pg, slot, 2) = h;
}

// Place an atom (fixed-point coordinates c, real = true) or a padding slot (far from everything:
// 16 A apart along x beyond 5000 A) and clear its accumulators for a new evaluation
__device__ __forceinline__ void placeSlot(const DevSynthesis &d, const UnitSmem &s, int slot,
                                          bool real, long long cx, long long cy, long long cz) {
  const float4 prm = s.prm[slot];
  float3 hi = make_float3(5000.0f + 16.0f * static_cast<float>(slot), 0.0f, 0.0f);
  float3 lo = make_float3(0.0f, 0.0f, 0.0f);
  if (real) {
    splitCoordinate(static_cast<double>(cx) * d.inv_gpos_scale, &hi.x, &lo.x);
    splitCoordinate(static_cast<double>(cy) * d.inv_gpos_scale, &hi.y, &lo.y);
    splitCoordinate(static_cast<double>(cz) * d.inv_gpos_scale, &hi.z, &lo.z);
  }
  // pass 1 payload: s * rho and rho
  putSlot(s, slot, hi, lo, prm.w, prm.z, 1.0f, 0.0f);
  s.fx[slot] = 0;
  s.fy[slot] = 0;
  s.fz[slot] = 0;
  s.fxo[slot] = 0;
  s.fyo[slot] = 0;
  s.fzo[slot] = 0;
  s.psi[slot] = 0;
  s.psio[slot] = 0;
  s.de[slot] = 0;
  s.deo[slot] = 0;
}

// All requested terms of a staged unit: coordinates, parameters and cleared accumulators in
// shared memory on entry (and a barrier since); forces in s.fx.. and per-molecule energies in
// s.nrg on exit, after a barrier.  WS: also write the GB workspace (psi, effective radii, dE/dR)
// to global memory.  CLASH: Coulomb and Lennard-Jones pairs, 1-4 pairs included, take the
// softened cores of s.clash (per unit molecule, zero for none, set before that barrier).  NECK:
// the neck GB term (s.neck holds the slots' neck indices).
template <bool FORCE, bool ENERGY, int TERMS, bool WS, bool CLASH = false, bool NECK = false,
          class Team>
__device__ void evaluateStaged(const DevSynthesis &d, const UnitSmem &s, const UnitShape &us,
                               const Team &team) {
  constexpr bool VALE = (TERMS & 1) != 0;
  constexpr bool NB = (TERMS & 2) != 0;
  const bool gb = ((TERMS & 4) != 0) && (d.igb != 0);
  const int nsys_u = us.nsys;
  const int nslots = us.nslots;
  const int ntiles = us.ntiles;

  // valence terms and GB pass 1 touch disjoint accumulators: no barrier between them
  if (VALE) {
    valenceTerms<FORCE, ENERGY, SmemValence, CLASH>(
        d, SmemValence(s, nsys_u, team.warp(), team.warps()));
    if (!gb) {
      team.sync();
    }
  }
  if (gb) {
    const int dealt = VALE ? unitMeta(s, kMetaBondChunk, nsys_u) +
                             unitMeta(s, kMetaAnglChunk, nsys_u) +
                             unitMeta(s, kMetaDiheChunk, nsys_u) : 0;
    gbRadiiTiles<FORCE, NECK>(d, s, nsys_u, ntiles, us.tile_base,
                              dealFrom(team.warp(), team.warps(), dealt), team.warps());
    team.sync();
    // effective radii, self terms (nonbonded_potential.tpp:730-805); a warp's 32 slots
    // belong to one molecule, so the self energies reduce across the warp
    const float inv_ps = 1.0f / static_cast<float>(1 << kPsiBits);
    const float ds = static_cast<float>(1 << kDeijdaBits);
    for (int slot = team.rank(); slot < nslots; slot += team.size()) {
      const int k = findOwner(s.slot0, nsys_u, slot);
      const int a = slot - s.slot0[k];
      float e_self = 0.0f;
      const float4 prm = s.prm[slot];
      float egbi = 1.0f;
      if (a < s.natom[k]) {
        const int gi = unitMeta(s, kMetaAtom0, k) + a;
        const double psi = static_cast<double>(int63ToLong(s.psi[slot], s.psio[slot])) *
                           static_cast<double>(inv_ps);
        egbi = effectiveRadius(d, gi, psi);
        float self_de;
        e_self = gbSelfTerm(d, prm.x, egbi, &self_de);
        if (FORCE) {
          atomicAddInt63(self_de * ds, &s.de[slot], &s.deo[slot]);
        }
        if (WS) {
          d.born_radii[gi] = egbi;
          d.psi[gi] = __double2ll_rn(static_cast<double>(psi) * d.psi_out_scale);
          d.psi_ovrf[gi] = 0;
        }
      }
      // pass 2 payload: charge (zero for padding, as prm.x is) and effective radius, and the
      // reciprocal radius beside the Lennard-Jones code
      slotValue(s.pb, slot, 2) = prm.x;
      slotValue(s.pd, slot, 2) = egbi;
      slotValue(s.pg, slot, 0) = 1.0f / egbi;
      slotValue(s.pg, slot, 2) = prm.y;
      if (ENERGY) {
        warpEnergy(s, k, kGb, e_self, d.nrg_scale);
      }
    }
    team.sync();
  }
  else if (NB) {
    // pass 2 payload for Coulomb / Lennard-Jones alone: charge in w1
    for (int slot = team.rank(); slot < nslots; slot += team.size()) {
      const float4 prm = s.prm[slot];
      slotValue(s.pb, slot, 2) = prm.x;
      slotValue(s.pg, slot, 2) = prm.y;     // the Lennard-Jones code, where pass 2 reads it
    }
    team.sync();
  }
  if (NB || gb) {
    if (NB && gb) {
      pairTiles<FORCE, ENERGY, true, true, CLASH>(d, s, nsys_u, ntiles, team.warp(),
                                                  team.warps());
    }
    else if (NB) {
      pairTiles<FORCE, ENERGY, true, false, CLASH>(d, s, nsys_u, ntiles, team.warp(),
                                                   team.warps());
    }
    else {
      pairTiles<FORCE, ENERGY, false, true>(d, s, nsys_u, ntiles, team.warp(), team.warps());
    }
    team.sync();
  }
  if (gb && FORCE) {
    // chain-rule prefactor of the OBC radii (nonbonded_potential.tpp:982-1021), and the
    // pass 3 payloads
    const float inv_ds = 1.0f / static_cast<float>(1 << kDeijdaBits);
    const float inv_ps = 1.0f / static_cast<float>(1 << kPsiBits);
    for (int slot = team.rank(); slot < nslots; slot += team.size()) {
      const int k = findOwner(s.slot0, nsys_u, slot);
      const int a = slot - s.slot0[k];
      float sde = 0.0f;
      if (a < s.natom[k]) {
        const int gi = unitMeta(s, kMetaAtom0, k) + a;
        sde = static_cast<float>(int63ToLong(s.de[slot], s.deo[slot])) * inv_ds;
        if (d.igb != 1) {
          const double psi = static_cast<double>(int63ToLong(s.psi[slot], s.psio[slot])) *
                             static_cast<double>(inv_ps);
          sde *= obcChainFactor(d, gi, psi);
        }
        if (WS) {
          d.sumdeijda[gi] = __double2ll_rn(static_cast<double>(sde) * d.psi_out_scale);
          d.sumdeijda_ovrf[gi] = 0;
        }
      }
      // pass 3 takes the separations and dE/dR alone
      slotValue(s.pg, slot, 2) = sde;
    }
    team.sync();
    gbDerivativeTiles(d, s, nsys_u, ntiles, us.tile_base, team.warp(), team.warps());
    team.sync();
  }
}

}  // namespace

}  // namespace sb

#endif