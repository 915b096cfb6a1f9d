// vlsg_rates.cuh -- per-active-point rates of one forward-Euler stage.
//
// Restates, per active point (defined, |phi| <= 0.5, lsAdvect.hpp:498):
//   the material choice and stop chain of integrateTime (lsAdvect.hpp:505-592),
//   the schemes' operator() -- EngquistOsher (lsEngquistOsher.hpp:42-162),
//   LaxFriedrichs (lsLaxFriedrichs.hpp:236-348), LocalLocalLaxFriedrichs
//   (lsLocalLocalLaxFriedrichs.hpp:298-421), LocalLaxFriedrichs
//   (lsLocalLaxFriedrichs.hpp:65-241), WENO3/5 (lsWENO.hpp:53-160 with
//   lsFiniteDifferences.hpp:58-123) -- and findGlobalAlphas
//   (lsAdvect.hpp:90-195), plus the per-point update of updateLevelSet
//   (lsAdvect.hpp:725-777).
// Expressions keep the reference's evaluation order; the library is compiled
// with -fmad=false so FP64 results are bit-identical to the CPU restatement.
//
// A block works on tiles of bricks (as the band passes, vlsg_frontier.cuh):
// its warps find the bricks' active cells, one list takes them all, and every
// thread evaluates points of the list.  Stencil values come through the slot's
// 27-neighbour table; points whose stencil reaches cells a boundary remaps go
// through the boundary mapping.  Outputs are compact over the active points:
// each tile reserves one entry per active cell, in the order of its list (brick
// by brick, cells ascending), and the value update finds a brick's entries
// from its first one (entry r of chain entry j at j * rateCap + r).
// Bound by the issue of the scheme's arithmetic and by load latency.  A warp
// per brick (about 45 active points in two rounds of 32, the second a third
// full) -> tiles, one B200: WENO5 FP32, 8.0M active points, 0.97 -> 0.80 ms; FP64,
// 0.9M points, 0.285 -> 0.24 ms; local Lax-Friedrichs FP64 on 18.5k points 137 ->
// 88 us, with reflective walls 390 -> 215 us (before the box normals below).
#pragma once

#include <type_traits>

#include "vlsg_common.cuh"
#include "vlsg_frontier.cuh"
#include "vlsg_passes.cuh"

namespace vlsg {
namespace { // internal linkage: every compilation unit has its own copy

constexpr int RATE_THREADS = 256;

template <class T> __device__ inline T sqr(T v) { return v * v; }
template <class T> __device__ inline T stdMax(T a, T b) { return (a < b) ? b : a; }
template <class T> __device__ inline T stdMin(T a, T b) { return (b < a) ? b : a; }

// Terms of material m that can be non-zero: bit k linear, 3 + k absolute,
// 6 + k square.
template <class T> __device__ inline unsigned velocityTerms(const vlsg_velocity_desc &v, int m) {
  unsigned bits = 0;
  for (int k = 0; k < 3; ++k) {
    if (T(v.lin_pos[m][k]) != T(0) || T(v.lin_neg[m][k]) != T(0)) bits |= 1u << k;
    if (T(v.abs_pos[m][k]) != T(0) || T(v.abs_neg[m][k]) != T(0)) bits |= 8u << k;
    if (T(v.sq_pos[m][k]) != T(0) || T(v.sq_neg[m][k]) != T(0)) bits |= 64u << k;
  }
  return bits;
}

// vlsg_velocity_desc evaluated term by term (order fixed by vlsg.h); terms:
// velocityTerms of the materials.  Most fields have a rate and a term or two,
// and the box schemes evaluate them 28 times a point: skipping a term costs a
// bit test instead of a load, a conversion from double and a compare.
template <class T>
__device__ inline T scalarVelocity(const vlsg_velocity_desc &v, const uint16_t *terms, int material,
                                   const T n[3]) {
  int m = material < v.n_materials ? material : v.n_materials - 1;
  if (m < 0) m = 0;
  const unsigned bits = terms[m];
  T s = T(v.rate[m]);
  if (bits == 0u) return s;
  for (int k = 0; k < 3; ++k) {
    if (!((bits >> k) & 1u)) continue;
    const T c = T(n[k] > 0 ? v.lin_pos[m][k] : v.lin_neg[m][k]);
    if (c != T(0)) s = s + c * n[k];
  }
  for (int k = 0; k < 3; ++k) {
    if (!((bits >> (3 + k)) & 1u)) continue;
    const T c = T(n[k] > 0 ? v.abs_pos[m][k] : v.abs_neg[m][k]);
    if (c != T(0)) s = s + c * fabs(n[k]);
  }
  for (int k = 0; k < 3; ++k) {
    if (!((bits >> (6 + k)) & 1u)) continue;
    const T c = T(n[k] > 0 ? v.sq_pos[m][k] : v.sq_neg[m][k]);
    if (c != T(0)) s = s + c * (n[k] * n[k]);
  }
  return s;
}
template <class T>
__device__ inline void vectorVelocity(const vlsg_velocity_desc &v, int material,
                                      T out[3]) {
  int m = material < v.n_materials ? material : v.n_materials - 1;
  if (m < 0) m = 0;
  for (int k = 0; k < 3; ++k) out[k] = T(v.vec[m][k]);
}

// Velocity of one evaluation site of an active point (site 0: the point
// itself; LocalLaxFriedrichs site 1 + q: box neighbour q, x fastest).
// FunctorVel evaluates the device functor; TableVel reads what the host
// callback returned for this point (entry material * sites + site).
// alpha(dir, material, cd, q): getDissipationAlpha at box neighbour q
// (LocalLaxFriedrichsAnalytical).
struct FunctorVel {
  const vlsg_velocity_desc &d;
  const uint16_t *terms;
  template <class T>
  __device__ void get(int material, const T n[3], int site, T &sv, T vv[3]) const {
    (void)site;
    sv = scalarVelocity<T>(d, terms, material, n);
    vectorVelocity<T>(d, material, vv);
  }
  template <class T> __device__ T alpha(int dir, int material, const T cd[3], int q) const {
    (void)cd, (void)q;
    int m = material < d.n_materials ? material : d.n_materials - 1;
    if (m < 0) m = 0;
    return T(d.alpha[m][dir]);
  }
};
struct TableVel {
  const double *s, *v;
  size_t base;
  int sites;
  const double *a; // alphas: ((p * L + material) * 27 + q) * 3 + dir, or none
  size_t alphaBase;
  // StencilLocalLaxFriedrichs: sites 28.. (nudged normals, scalar only) at
  // (p * L + material) * 162 + site - 28
  const double *s2;
  size_t base2;
  template <class T>
  __device__ void get(int material, const T n[3], int site, T &sv, T vv[3]) const {
    (void)n;
    if (site >= 28) {
      sv = T(s2[base2 + (size_t)material * 162 + (site - 28)]);
      vv[0] = vv[1] = vv[2] = T(0);
      return;
    }
    const size_t i = base + (size_t)material * sites + site;
    sv = T(s[i]);
    for (int k = 0; k < 3; ++k) vv[k] = T(v[3 * i + k]);
  }
  template <class T> __device__ T alpha(int dir, int material, const T cd[3], int q) const {
    (void)cd;
    return a ? T(a[alphaBase + ((size_t)material * 27 + q) * 3 + dir]) : T(0);
  }
};

template <class T> struct RateArgs {
  GridDev g;
  MapView m;
  Buf<T> ls[VLSG_MAX_LEVEL_SETS];
  int L;
  const int *slotList, *nSlots;
  const int *nbr;       // 27-neighbour table per slot
  const uint8_t *cflag; // CF_* per slot
  const uint64_t *def;  // defined masks of the top level set
  const uint8_t *visit; // its bricks that may hold a defined cell, or null: any
  uint64_t *act;        // out: active masks of the top level set
  int scheme;
  double cfl;
  double dissipationAlpha;
  int calcNormals;
  int adaptive;
  double adaptiveFactor;
  int checkDiss;
  T globalAlpha[3];
  // outputs, compact over the active points: a brick reserves one entry per
  // active cell (rateNext) and records where they start (rateBase[slot]);
  // chain entry j of entry r is at j * rateCap + r, in the order of the
  // brick's active cells
  T *rateV;
  T *rateStop;
  T *rateD; // the dissipation per chain entry (setSaveAdvectionVelocities), or null
  uint8_t *rateLen;
  size_t rateCap;
  unsigned long long *rateNext;
  unsigned long long *rateBase;
  int rateOverflowErr; // err bit for a brick left out (0: the host checks rateNext)
  unsigned long long *minStep;  // complement of the smallest non-negative step's bits
  unsigned long long *alphaMax; // bits of the LLF/LLLF alphas
  unsigned long long *counts;   // out: active cells, band cells
  int *err;
  // host callback mode: active points before list entry w, and the
  // velocities of point p at (p * L + material) * velSites + site
  const uint32_t *actOff;
  const double *velS, *velV;
  int velSites;
  const double *alphaTab; // LocalLaxFriedrichsAnalytical: the alpha callback's answers
  const double *velS2;    // StencilLocalLaxFriedrichs: the nudged-normal answers
  // StencilLocalLaxFriedrichs: baseNormalEpsilon, the dissipation limit, and
  // per warp the last (HRLE order) call's finalAlphas: key, alphas
  double sllfEps;
  double maxDissipation;
  unsigned long long *sllfKey;
  double *sllfAlpha;
  // setIgnoreVoids: void bits of the top level set (no rates there), or none
  const uint64_t *voidMask;
  // sharding: only points with z in [ownLo, ownHi) count towards the time
  // step, the alphas and the point updates (ownZ false: every point)
  bool ownZ;
  int ownLo, ownHi;
  // batching form (slotDom non-null): per slot its domain; per domain its
  // gridDelta and velocity functor, and this pass's reductions (RED_* words
  // per domain: smallest step bits, alpha bits x3, active cells) in place of
  // minStep / alphaMax / counts
  const int *slotDom;
  const double *domDelta;
  const vlsg_velocity_desc *domVel;
  unsigned long long *domRed;
};
constexpr int RED_MIN = 0, RED_ALPHA = 1, RED_ACTIVE = 4, RED_WORDS = 5;

// Reader of the top level set around one active point near a boundary that
// remaps cells: cells of the grid through the slot's 27-neighbour table
// (offsets up to 8 cells), the others through the boundary mapping.
template <class T> struct Stencil {
  const GridDev &g;
  const MapView &m;
  const Buf<T> &b;
  const int *nb27;
  int lx, ly, lz, x0, y0, z0;
  __device__ T at(int dx, int dy, int dz) const {
    const int nx = lx + dx, ny = ly + dy, nz = lz + dz;
    if (!cellExists(g, x0 + nx, y0 + ny, z0 + nz))
      return cellValueRaw<T>(g, m, b, x0 + nx, y0 + ny, z0 + nz);
    const int ref = nb27[((nz >> 3) + 1) * 9 + ((ny >> 3) + 1) * 3 + ((nx >> 3) + 1)];
    if (ref < 0) return b.farSign[-1 - ref] < 0 ? Lim<T>::lowest() : Lim<T>::max();
    return b.vals[(size_t)ref * BV + ((nz & 7) * 64 + (ny & 7) * 8 + (nx & 7))];
  }
  __device__ T axis(int d, int off) const {
    return d == 0 ? at(off, 0, 0) : (d == 1 ? at(0, off, 0) : at(0, 0, off));
  }
};

// Reader of the top level set around one active point through the slot's
// 27-neighbour table (offsets up to 8 cells; every cell it reaches exists and
// is not remapped by a boundary).
template <class T> struct TableStencil {
  const T *vals;
  const int8_t *farSign;
  const int *nb27;
  int lx, ly, lz;
  __device__ T at(int dx, int dy, int dz) const {
    const int nx = lx + dx, ny = ly + dy, nz = lz + dz;
    const int ref = nb27[((nz >> 3) + 1) * 9 + ((ny >> 3) + 1) * 3 + ((nx >> 3) + 1)];
    if (ref < 0) return farSign[-1 - ref] < 0 ? Lim<T>::lowest() : Lim<T>::max();
    return vals[(size_t)ref * BV + ((nz & 7) * 64 + (ny & 7) * 8 + (nx & 7))];
  }
  __device__ T axis(int d, int off) const {
    return d == 0 ? at(off, 0, 0) : (d == 1 ? at(0, off, 0) : at(0, 0, off));
  }
};

template <class T, class St>
__device__ inline void oneSided(const St &S, int i, T phi0, T gridDelta,
                                int order, T &diffPos, T &diffNeg) {
  const T deltaPos = gridDelta;
  const T deltaNeg = -gridDelta;
  const T phiPos = S.axis(i, 1);
  const T phiNeg = S.axis(i, -1);
  diffPos = (phiPos - phi0) / deltaPos;
  diffNeg = (phiNeg - phi0) / deltaNeg;
  if (order == 2) {
    const T deltaPosPos = 2 * gridDelta;
    const T deltaNegNeg = -2 * gridDelta;
    const T phiPosPos = S.axis(i, 2);
    const T phiNegNeg = S.axis(i, -2);
    const T diff00 =
        (((deltaNeg * phiPos - deltaPos * phiNeg) / (deltaPos - deltaNeg) + phi0)) /
        (deltaPos * deltaNeg);
    const T diffNegNeg = (((deltaNeg * phiNegNeg - deltaNegNeg * phiNeg) /
                               (deltaNegNeg - deltaNeg) +
                           phi0)) /
                         (deltaNegNeg * deltaNeg);
    const T diffPosPos = (((deltaPos * phiPosPos - deltaPosPos * phiPos) /
                               (deltaPosPos - deltaPos) +
                           phi0)) /
                         (deltaPosPos * deltaPos);
    if (signbit(diff00) == signbit(diffPosPos)) {
      if (fabs(diffPosPos * deltaPos) < fabs(diff00 * deltaNeg))
        diffPos -= deltaPos * diffPosPos;
      else
        diffPos += deltaNeg * diff00;
    }
    if (signbit(diff00) == signbit(diffNegNeg)) {
      if (fabs(diffNegNeg * deltaNeg) < fabs(diff00 * deltaPos))
        diffNeg -= deltaNeg * diffNegNeg;
      else
        diffNeg += deltaPos * diff00;
    }
  }
}

template <class T>
__device__ inline T weno3(const T *x, T delta, bool plus) {
  const T eps = T(1e-6);
  T d0, d1, d2;
  if (plus) {
    d0 = x[2] - x[1];
    d1 = x[3] - x[2];
    d2 = x[4] - x[3];
    const T N = eps + sqr(d2 - d1);
    const T Dd = eps + sqr(d1 - d0);
    const T D2 = Dd * Dd;
    const T wp = D2 / (D2 + 2 * N * N);
    return (d0 + d1 - wp * (d2 - 2 * d1 + d0)) / (2 * delta);
  }
  d0 = x[1] - x[0];
  d1 = x[2] - x[1];
  d2 = x[3] - x[2];
  const T N = eps + sqr(d1 - d0);
  const T Dd = eps + sqr(d2 - d1);
  const T D2 = Dd * Dd;
  const T wp = D2 / (D2 + 2 * N * N);
  return (d1 + d2 - wp * (d0 - 2 * d1 + d2)) / (2 * delta);
}

template <class T>
__device__ inline T weno5(const T *x, T dx, bool plus) {
  const T eps = T(1e-6);
  T d[5];
  if (!plus) {
#pragma unroll
    for (int i = 0; i < 5; ++i) d[i] = x[i + 1] - x[i];
  } else {
#pragma unroll
    for (int i = 0; i < 5; ++i) d[i] = x[6 - i] - x[5 - i];
  }
  const T c1312 = T(13.0 / 12.0), c14 = T(1.0 / 4.0), c16 = T(1.0 / 6.0);
  const T s1 = c1312 * sqr(d[0] - 2 * d[1] + d[2]) + c14 * sqr(d[0] - 4 * d[1] + 3 * d[2]);
  const T s2 = c1312 * sqr(d[1] - 2 * d[2] + d[3]) + c14 * sqr(d[1] - d[3]);
  const T s3 = c1312 * sqr(d[2] - 2 * d[3] + d[4]) + c14 * sqr(3 * d[2] - 4 * d[3] + d[4]);
  const T eps_scaled = eps * dx * dx;
  const T al1 = T(0.1) / (eps_scaled + s1);
  const T al2 = T(0.6) / (eps_scaled + s2);
  const T al3 = T(0.3) / (eps_scaled + s3);
  const T alsum = al1 + al2 + al3;
  const T p1 = c16 * (2 * d[0] - 7 * d[1] + 11 * d[2]);
  const T p2 = c16 * (-d[1] + 5 * d[2] + 2 * d[3]);
  const T p3 = c16 * (2 * d[2] + 5 * d[3] - d[4]);
  return (al1 * p1 + al2 * p2 + al3 * p3) / (alsum * dx);
}

// The normal LocalLaxFriedrichs takes at offset (ox, oy, oz)
// (lsLocalLaxFriedrichs.hpp:194-212).
template <class T, class St>
__device__ inline void boxNormal(const St &S, T gridDelta, int ox, int oy, int oz, T normal[3]) {
  T nm = 0.;
  const T center = S.at(ox, oy, oz);
  for (int dir = 0; dir < 3; ++dir) {
    const T neg = S.at(ox - (dir == 0), oy - (dir == 1), oz - (dir == 2));
    const T pos = S.at(ox + (dir == 0), oy + (dir == 1), oz + (dir == 2));
    const T dPos = (pos - center) / gridDelta;
    const T dNeg = (center - neg) / gridDelta;
    normal[dir] = (dPos + dNeg) * T(0.5);
    nm += normal[dir] * normal[dir];
  }
  nm = T(1.) / sqrt(nm);
  for (int dir = 0; dir < 3; ++dir) normal[dir] *= nm;
}

// Central differences at box neighbour q (x fastest):
// calculateNormalComponent of lsLocalLaxFriedrichsAnalytical.hpp:30-34.
template <class T, class St>
__device__ inline void boxDifferences(const St &S, T gridDelta, int q, T cd[3]) {
  const int ox = q % 3 - 1, oy = (q / 3) % 3 - 1, oz = q / 9 - 1;
  const T center = S.at(ox, oy, oz);
  for (int dir = 0; dir < 3; ++dir) {
    const T neg = S.at(ox - (dir == 0), oy - (dir == 1), oz - (dir == 2));
    const T pos = S.at(ox + (dir == 0), oy + (dir == 1), oz + (dir == 2));
    const T diffPos = (pos - center) / gridDelta;
    const T diffNeg = (center - neg) / gridDelta;
    cd[dir] = (diffPos + diffNeg) * T(0.5);
  }
}

// StencilLocalLaxFriedrichsScalar's FIRST_ORDER gradient component i at
// box offset (ox, oy, oz): the three values along i are taken with
// coordinate i set to -1, 0, 1 whatever the offset's (calculateGradient /
// calculateNormal, lsStencilLocalLaxFriedrichsScalar.hpp:336-378;
// FiniteDifferences, lsFiniteDifferences.hpp:132-181).
template <class T, class St>
__device__ inline T sllfGrad(const St &S, double delta, int ox, int oy, int oz, int i) {
  T v[3];
  for (int j = 0; j < 3; ++j)
    v[j] = S.at(i == 0 ? j - 1 : ox, i == 1 ? j - 1 : oy, i == 2 ? j - 1 : oz);
  const T dNeg = T((v[1] - v[0]) / delta);
  const T dPos = T((v[2] - v[1]) / delta);
  return T((dPos + dNeg) * 0.5);
}
template <class T, class St>
__device__ inline void sllfNormal(const St &S, double delta, int ox, int oy, int oz, T n[3]) {
  T modulus = 0.;
  for (int i = 0; i < 3; ++i) {
    n[i] = sllfGrad<T>(S, delta, ox, oy, oz, i);
    modulus += n[i] * n[i];
  }
  modulus = T(1) / sqrt(modulus);
  for (int i = 0; i < 3; ++i) n[i] *= modulus;
}
// calculateSimpleAdaptiveEpsilon (ADAPTIVE_EPSILON_STRATEGY 1, :60-75)
template <class T> __device__ inline T sllfEpsilon(T velocity, double baseNormalEpsilon, double delta) {
  const T absVel = fabs(velocity);
  const T baseEps = T(baseNormalEpsilon * delta);
  if (absVel > T(1e-10)) {
    const T scale = stdMax(T(0.1), stdMin(T(10.0), absVel));
    return baseEps * scale;
  }
  return baseEps;
}

// StencilLocalLaxFriedrichsScalar<T,3,1>::operator() (:219-400).  Velocity
// sites: 0 the point, 1 + q the stencil point q (x fastest), 28 + 6q + 2k
// (+1) the normal of q nudged by -DN (+DN) along k.  alphas[0..2] receive
// this call's finalAlphas and alphas[3] = 1 when the call gets past the
// zero-velocity return.
template <class T, class St, class Vel>
__device__ void evalStencilLLF(const RateArgs<T> &A, const Vel &vel, const St &S, int material,
                               T *alphas, T &outG, T &outD) {
  const double delta = A.g.delta;
  T normalVector[3];
  sllfNormal<T>(S, delta, 0, 0, 0, normalVector);
  T sv0, vv0[3];
  vel.get(material, normalVector, 0, sv0, vv0);
  double scalarVelocity = (double)sv0;
  for (int i = 0; i < 3; ++i) scalarVelocity += (double)(vv0[i] * normalVector[i]);
  if (scalarVelocity == 0.) {
    outG = 0;
    outD = 0;
    return;
  }
  T gradSq = 0;
  for (int i = 0; i < 3; ++i) {
    const T gi = sllfGrad<T>(S, delta, 0, 0, 0, i);
    gradSq += gi * gi;
  }
  const T hamiltonian = T((double)sqrt(gradSq) * scalarVelocity);
  T maxAlpha[3] = {0, 0, 0};
  // D = 2 (the plane of a z-periodic grid): the 3x3 stencil of the plane and
  // the normal nudged in x and y only, as the 2D reference does; the z terms
  // below then add exact zeros
  const bool planar = A.g.planar != 0;
  const int nSt = planar ? 9 : 27, nDir = planar ? 2 : 3;
  int cx = -1, cy = -1, cz = planar ? 0 : -1;
  for (int st = 0; st < nSt; ++st) {
    T ln[3];
    sllfNormal<T>(S, delta, cx, cy, cz, ln);
    // a corrupted normal leaves the stencil index where it is (:288-293)
    if (fabs(ln[0]) < T(1e-6) && fabs(ln[1]) < T(1e-6) && fabs(ln[2]) < T(1e-6)) continue;
    const int q = (cz + 1) * 9 + (cy + 1) * 3 + (cx + 1);
    T lsv, lvv[3];
    vel.get(material, ln, 1 + q, lsv, lvv);
    for (int dir = 0; dir < 3; ++dir) lsv += lvv[dir] * ln[dir];
    const T DN = sllfEpsilon<T>(lsv, A.sllfEps, delta);
    T np[3] = {ln[0], ln[1], ln[2]}, nn[3] = {ln[0], ln[1], ln[2]}, vd[3] = {0, 0, 0};
    for (int k = 0; k < nDir; ++k) {
      np[k] -= DN;
      nn[k] += DN;
      T vp, vn, unused[3];
      vel.get(material, np, 28 + 6 * q + 2 * k, vp, unused);
      vel.get(material, nn, 28 + 6 * q + 2 * k + 1, vn, unused);
      vd[k] = T((double)(vn - vp) / (2.0 * (double)DN));
      np[k] += DN;
      nn[k] -= DN;
    }
    T gr[3];
    for (int i = 0; i < 3; ++i) gr[i] = sllfGrad<T>(S, delta, cx, cy, cz, i);
    T denom = 0;
    for (int i = 0; i < 3; ++i) denom += gr[i] * gr[i];
    for (int k = 0; k < 3; ++k) {
      T monti = 0, toifl = 0;
      for (int j = 0; j < 2; ++j) {
        const int idx = (k + 1 + j) % 3;
        monti += gr[idx] * gr[idx];
        toifl += gr[idx] * vd[idx];
      }
      monti *= vd[k] / denom;
      toifl *= -gr[k] / denom;
      const T osher = lsv * ln[k];
      maxAlpha[k] = stdMax(maxAlpha[k], T(fabs(monti + toifl + osher)));
    }
    // incrementIndex, x fastest (:196-204)
    if (cx < 1) {
      ++cx;
    } else {
      cx = -1;
      if (cy < 1) {
        ++cy;
      } else {
        cy = -1;
        ++cz;
      }
    }
  }
  T dissipation = 0.;
  for (int d = 0; d < 3; ++d) {
    T v[3];
    for (int j = 0; j < 3; ++j) v[j] = S.at(d == 0 ? j - 1 : 0, d == 1 ? j - 1 : 0, d == 2 ? j - 1 : 0);
    const T dNeg = T((v[1] - v[0]) / delta);
    const T dPos = T((v[2] - v[1]) / delta);
    const T gradientDiff = T((dPos - dNeg) * 0.5);
    const T finalAlpha = stdMin(maxAlpha[d], T(A.maxDissipation));
    alphas[d] = finalAlpha;
    dissipation += finalAlpha * gradientDiff;
  }
  alphas[3] = T(1);
  outG = hamiltonian;
  outD = dissipation;
}

// One scheme evaluation (Hamiltonian, dissipation) for `material`.
// Scheme families a rate kernel is compiled for: every scheme but the
// stencil one (chosen at run time), WENO only, StencilLocalLaxFriedrichs only,
// LocalLaxFriedrichs 1st and 2nd order with the normals of the box cells
// computed once per cell (`box`: component d at BOX_CELLS * d around the
// point's own, x fastest, edge BOX_EDGE).
enum : int { FAM_ANY = 0, FAM_WENO = 1, FAM_STENCIL = 2, FAM_BOX = 3 };
constexpr int BOX_EDGE = BS + 2, BOX_CELLS = BOX_EDGE * BOX_EDGE * BOX_EDGE;

template <class T, class St, class Vel, int FAM = FAM_ANY>
__device__ void evalScheme(const RateArgs<T> &A, const Vel &vel,
                           const St &S, T C, int material, T *alphas,
                           T &outG, T &outD, double delta, const T *box) {
  if constexpr (FAM == FAM_STENCIL) {
    (void)C;
    evalStencilLLF<T>(A, vel, S, material, alphas, outG, outD);
    return;
  }
  const T gridDelta = T(delta);
  const int sch = A.scheme;
  if (FAM == FAM_WENO ||
      (FAM == FAM_ANY && (sch == VLSG_WENO_3RD_ORDER || sch == VLSG_WENO_5TH_ORDER))) {
    const int r = sch == VLSG_WENO_3RD_ORDER ? 2 : 3;
    T gradPosTotal = 0, gradNegTotal = 0;
    T wMinus[3], wPlus[3], st[7], phiPos[3], phiNeg[3];
    for (int i = 0; i < 3; i++) {
      st[r] = C;
      for (int k = 1; k <= r; ++k) {
        st[r + k] = S.axis(i, k);
        st[r - k] = S.axis(i, -k);
      }
      phiPos[i] = st[r + 1], phiNeg[i] = st[r - 1];
      if (r == 2) {
        wMinus[i] = weno3<T>(st, gridDelta, false);
        wPlus[i] = weno3<T>(st, gridDelta, true);
      } else {
        wMinus[i] = weno5<T>(st, gridDelta, false);
        wPlus[i] = weno5<T>(st, gridDelta, true);
      }
      gradPosTotal += sqr(stdMax(wMinus[i], T(0))) + sqr(stdMin(wPlus[i], T(0)));
      gradNegTotal += sqr(stdMin(wMinus[i], T(0))) + sqr(stdMax(wPlus[i], T(0)));
    }
    T vel_grad = 0.;
    T n[3] = {0, 0, 0};
    // the scheme receives dissipationAlpha as its calcNormal flag
    if (A.dissipationAlpha != 0.0) {
      T denominator = 0;
      for (int i = 0; i < 3; i++) {
        n[i] = phiPos[i] - phiNeg[i];
        denominator += n[i] * n[i];
      }
      if (denominator > 0) {
        denominator = T(1.) / sqrt(denominator);
        for (int i = 0; i < 3; ++i) n[i] *= denominator;
      }
    }
    T sv, vv[3];
    vel.get(material, n, 0, sv, vv);
    if (sv > 0)
      vel_grad += sqrt(gradPosTotal) * sv;
    else
      vel_grad += sqrt(gradNegTotal) * sv;
    for (int w = 0; w < 3; w++) {
      if (vv[w] > T(0))
        vel_grad += vv[w] * wMinus[w];
      else
        vel_grad += vv[w] * wPlus[w];
    }
    outG = vel_grad;
    outD = 0;
    return;
  }
  if constexpr (FAM == FAM_WENO) {
    return;
  } else {
  const int order = (sch == VLSG_ENGQUIST_OSHER_2ND_ORDER ||
                     sch == VLSG_LAX_FRIEDRICHS_2ND_ORDER ||
                     sch == VLSG_LOCAL_LOCAL_LAX_FRIEDRICHS_2ND_ORDER ||
                     sch == VLSG_LOCAL_LAX_FRIEDRICHS_2ND_ORDER)
                        ? 2
                        : 1;
  T gradPos[3], gradNeg[3];
  if (FAM == FAM_ANY &&
      (sch == VLSG_ENGQUIST_OSHER_1ST_ORDER || sch == VLSG_ENGQUIST_OSHER_2ND_ORDER)) {
    T gradPosTotal = 0, gradNegTotal = 0;
    for (int i = 0; i < 3; i++) {
      T diffPos, diffNeg;
      oneSided<T>(S, i, C, gridDelta, order, diffPos, diffNeg);
      gradPos[i] = diffNeg;
      gradNeg[i] = diffPos;
      gradPosTotal += sqr(stdMax(diffNeg, T(0))) + sqr(stdMin(diffPos, T(0)));
      gradNegTotal += sqr(stdMin(diffNeg, T(0))) + sqr(stdMax(diffPos, T(0)));
    }
    T vel_grad = 0.;
    T n[3] = {0, 0, 0};
    if (A.calcNormals) {
      T denominator = 0;
      for (int i = 0; i < 3; i++) {
        const T pos = S.axis(i, 1) - C;
        const T neg = C - S.axis(i, -1);
        n[i] = (pos + neg) * T(0.5);
        denominator += n[i] * n[i];
      }
      denominator = T(1.) / sqrt(denominator);
      for (int i = 0; i < 3; ++i) n[i] *= denominator;
    }
    T sv, vv[3];
    vel.get(material, n, 0, sv, vv);
    if (sv > 0)
      vel_grad += sqrt(gradPosTotal) * sv;
    else
      vel_grad += sqrt(gradNegTotal) * sv;
    for (int w = 0; w < 3; w++) {
      if (vv[w] > T(0))
        vel_grad += vv[w] * gradPos[w];
      else
        vel_grad += vv[w] * gradNeg[w];
    }
    outG = vel_grad;
    outD = 0;
    return;
  }
  const bool globalLF = FAM == FAM_ANY && (sch == VLSG_LAX_FRIEDRICHS_1ST_ORDER ||
                                           sch == VLSG_LAX_FRIEDRICHS_2ND_ORDER);
  const bool calcNormal = globalLF ? (A.calcNormals != 0) : true;
  const T alphaFactor = T(A.dissipationAlpha);
  T grad = 0., dissipation = 0.;
  T n[3] = {0, 0, 0};
  T normalModulus = 0;
  for (int i = 0; i < 3; i++) {
    T diffPos, diffNeg;
    oneSided<T>(S, i, C, gridDelta, order, diffPos, diffNeg);
    gradPos[i] = diffNeg;
    gradNeg[i] = diffPos;
    if (calcNormal) {
      n[i] = (diffNeg + diffPos) * T(0.5);
      normalModulus += n[i] * n[i];
    }
    grad += sqr((diffNeg + diffPos) * T(0.5));
    if (globalLF)
      dissipation += alphaFactor * A.globalAlpha[i] * (diffPos - diffNeg) * T(0.5);
  }
  if (calcNormal) {
    normalModulus = T(1.) / sqrt(normalModulus);
    for (int i = 0; i < 3; ++i) n[i] *= normalModulus;
  }
  T sv, vv[3];
  vel.get(material, n, 0, sv, vv);
  T totalGrad = 0.;
  if (sv != T(0)) totalGrad = sv * sqrt(grad);
  for (int w = 0; w < 3; w++) {
    if (vv[w] > T(0))
      totalGrad += vv[w] * gradPos[w];
    else
      totalGrad += vv[w] * gradNeg[w];
  }
  if (globalLF) {
    outG = totalGrad;
    outD = (totalGrad != T(0)) ? dissipation : T(0);
    return;
  }
  if (totalGrad == T(0)) {
    outG = 0;
    outD = 0;
    return;
  }
  if (FAM == FAM_ANY && sch == VLSG_LOCAL_LAX_FRIEDRICHS_ANALYTICAL_1ST_ORDER) {
    // the user's alphas over the 3x3x3 box at the central differences
    // (calculateNormalComponent, not normalised), no alphaFactor
    // (D = 2, the plane of a z-periodic grid: the plane's 3x3 box and the
    // directions x and y, as the 2D reference asks them)
    T alpha[3] = {0, 0, 0};
    const int q0 = A.g.planar ? 9 : 0, q1 = A.g.planar ? 18 : 27, nDir = A.g.planar ? 2 : 3;
    for (int q = q0; q < q1; ++q) {
      T cd[3];
      boxDifferences<T>(S, gridDelta, q, cd);
      for (int dir = 0; dir < nDir; ++dir) {
        const T tempAlpha = vel.alpha(dir, material, cd, q);
        alpha[dir] = stdMax(alpha[dir], tempAlpha);
        alphas[dir] = stdMax(alphas[dir], tempAlpha);
      }
    }
    for (int i = 0; i < 3; ++i) dissipation += alpha[i] * (gradNeg[i] - gradPos[i]) * T(0.5);
    outG = totalGrad;
    outD = dissipation;
    return;
  }
  if (FAM == FAM_ANY && (sch == VLSG_LOCAL_LOCAL_LAX_FRIEDRICHS_1ST_ORDER ||
                         sch == VLSG_LOCAL_LOCAL_LAX_FRIEDRICHS_2ND_ORDER)) {
    for (int i = 0; i < 3; ++i) {
      const T alpha = fabs((sv + vv[i]) * n[i]);
      alphas[i] = stdMax(alphas[i], alpha);
      dissipation += alphaFactor * alpha * (gradNeg[i] - gradPos[i]) * T(0.5);
    }
    outG = totalGrad;
    outD = dissipation;
    return;
  }
  // LocalLaxFriedrichs: alphas over the 3x3x3 box, x fastest (D = 2: the
  // plane's 3x3 box, q 9..17)
  T alpha[3] = {0, 0, 0};
  const auto take = [&](int q, const T normal[3]) {
    T scaVel, vecVel[3];
    vel.get(material, normal, 1 + q, scaVel, vecVel);
    for (int dir = 0; dir < 3; ++dir) {
      const T tempAlpha = fabs((scaVel + vecVel[dir]) * normal[dir]);
      alpha[dir] = stdMax(alpha[dir], tempAlpha);
      alphas[dir] = stdMax(alphas[dir], tempAlpha);
    }
  };
  if constexpr (FAM == FAM_BOX) {
#pragma unroll 1
    for (int row = 0; row < 9; ++row) {
      const T *at = box + (row / 3 - 1) * BOX_EDGE * BOX_EDGE + (row % 3 - 1) * BOX_EDGE;
#pragma unroll
      for (int ox = -1; ox <= 1; ++ox) {
        const T normal[3] = {at[ox], at[ox + BOX_CELLS], at[ox + 2 * BOX_CELLS]};
        take(3 * row + ox + 1, normal);
      }
    }
  } else {
    const int q1 = A.g.planar ? 18 : 27;
    for (int q = A.g.planar ? 9 : 0; q < q1; ++q) {
      T normal[3];
      boxNormal<T>(S, gridDelta, q % 3 - 1, (q / 3) % 3 - 1, q / 9 - 1, normal);
      take(q, normal);
    }
  }
  for (int i = 0; i < 3; ++i)
    dissipation += alphaFactor * alpha[i] * (gradNeg[i] - gradPos[i]) * T(0.5);
  outG = totalGrad;
  outD = dissipation;
  }
}

template <class T>
__device__ inline T lsValueAt(const Buf<T> &b, int slot, int c) {
  return b.vals[(size_t)slot * BV + c];
}

// Bits of a per-point step for the minimum (v >= 0; NaN or "no point" -1
// never lowers the minimum, lsAdvect.hpp:591) and of an alpha for the maximum.
__device__ inline unsigned long long stepBits(double v) {
  return (v >= 0.0) ? orderedBits(v + 0.0) : ~0ull;
}
__device__ inline unsigned long long alphaBits(double v) {
  return (v > 0.0) ? orderedBits(v) : 0ull;
}
__device__ inline unsigned long long warpMinU64(unsigned long long b) {
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long t = __shfl_xor_sync(0xffffffffu, b, o);
    b = t < b ? t : b;
  }
  return b;
}
__device__ inline unsigned long long warpMaxU64(unsigned long long b) {
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long t = __shfl_xor_sync(0xffffffffu, b, o);
    b = t > b ? t : b;
  }
  return b;
}

// integrateTime for one active point (lsAdvect.hpp:501-592): the material
// chain, the stored rates (velocity as updateLevelSet applies it,
// lsAdvect.hpp:738-744, and the stop value) and the point's time budget.
template <class T, class St, class Vel, int FAM = FAM_ANY>
__device__ inline double ratePoint(const RateArgs<T> &A, const Vel &vel,
                                   const St &S, int slot, int c, T C, T *alphas,
                                   double delta, size_t q, const T *box) {
  const int L = A.L;
  T value = C;
  double maxStepTime = 0;
  double cfl = A.cfl;
  int len = 0;
  const bool isVoid = A.voidMask && ((A.voidMask[(size_t)slot * 8 + (c >> 6)] >> (c & 63)) & 1ull);
  for (int cur = L - 1; cur >= 0; --cur) {
    T g = 0, d = 0;
    for (int lower = 0; lower < L && !isVoid; ++lower) {
      const T lv = lower == L - 1 ? C : lsValueAt<T>(A.ls[lower], slot, c);
      if ((double)lv <= (double)value + 1e-4) {
        evalScheme<T, St, Vel, FAM>(A, vel, S, C, lower, alphas, g, d, delta, box);
        break;
      }
    }
    const T velocity = g - d;
    T veff = velocity;
    if ((A.checkDiss && (g < 0 && velocity > 0)) || (g > 0 && velocity < 0)) veff = 0;
    T stop;
    bool done = true;
    if (velocity > 0.) {
      maxStepTime += cfl / velocity;
      stop = Lim<T>::lowest();
    } else if (velocity == 0.) {
      maxStepTime = (double)Lim<T>::max();
      stop = Lim<T>::max();
    } else {
      const T valueBelow = cur > 0 ? lsValueAt<T>(A.ls[cur - 1], slot, c) : Lim<T>::max();
      const T difference = fabs(valueBelow - value);
      if ((double)difference >= cfl) {
        maxStepTime -= cfl / velocity;
        stop = Lim<T>::max();
      } else if (A.adaptive && (double)difference > A.adaptiveFactor * cfl) {
        maxStepTime -= A.adaptiveFactor * cfl / velocity;
        stop = Lim<T>::max();
      } else {
        cfl -= difference;
        value = valueBelow;
        maxStepTime -= difference / velocity;
        stop = valueBelow;
        done = false;
      }
    }
    A.rateV[(size_t)len * A.rateCap + q] = veff;
    A.rateStop[(size_t)len * A.rateCap + q] = stop;
    if (A.rateD) A.rateD[(size_t)len * A.rateCap + q] = d;
    ++len;
    if (done) break;
  }
  A.rateLen[q] = (uint8_t)len;
  return maxStepTime;
}

// Cells around a point a scheme reads: WENO5 3 along each axis, the box
// schemes 2 (lsLocalLaxFriedrichs.hpp:194-212).
constexpr int STENCIL_REACH = 3;

// Stencil around local position (lx, ly, lz) of `slot` (up to one cell outside
// the brick): the table reader, or the mapping one where a cell within reach R
// is remapped by a boundary; fn(stencil).
template <class T, int R, class Fn>
__device__ inline void withStencilAt(const RateArgs<T> &A, int slot, int lx, int ly, int lz, Fn fn) {
  const Buf<T> &top = A.ls[A.L - 1];
  if (A.cflag[slot] & CF_NEAR) {
    int bx, by, bz;
    brickCoords(A.g, A.m.slotBrick[slot], bx, by, bz);
    const int x0 = A.g.org[0] + bx * BS, y0 = A.g.org[1] + by * BS, z0 = A.g.org[2] + bz * BS;
    // (the cells that exist form a box: its corners tell)
    if (!cellExists(A.g, x0 + lx - R, y0 + ly - R, z0 + lz - R) ||
        !cellExists(A.g, x0 + lx + R, y0 + ly + R, z0 + lz + R)) {
      const Stencil<T> S{A.g, A.m, top, A.nbr + (size_t)slot * 27, lx, ly, lz, x0, y0, z0};
      fn(S);
      return;
    }
  }
  const TableStencil<T> S{top.vals, top.farSign, A.nbr + (size_t)slot * 27, lx, ly, lz};
  fn(S);
}

// Stencil of local cell c of `slot`; fn(stencil, centre value).
template <class T, class Fn>
__device__ inline void withStencil(const RateArgs<T> &A, int slot, int c, Fn fn) {
  const T C = A.ls[A.L - 1].vals[(size_t)slot * BV + c];
  withStencilAt<T, STENCIL_REACH>(A, slot, c & 7, (c >> 3) & 7, c >> 6,
                                  [&](const auto &S) { fn(S, C); });
}

// Active mask of a brick (defined cells with |phi| <= 0.5, lsAdvect.hpp:498;
// lane z returns plane z): one coalesced read of the brick's 512 values.
template <class T>
__device__ inline uint64_t activePlanes(const T *vals, int slot) {
  const int lane = threadIdx.x & 31;
  const T *p = vals + (size_t)slot * BV + lane;
  T v[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = p[32 * i];
  uint64_t mine = 0;
#pragma unroll
  for (int z = 0; z < 8; ++z) {
    const unsigned lo = __ballot_sync(0xffffffffu, isDef(v[2 * z]) && fabs(v[2 * z]) <= T(0.5));
    const unsigned hi =
        __ballot_sync(0xffffffffu, isDef(v[2 * z + 1]) && fabs(v[2 * z + 1]) <= T(0.5));
    if (lane == z) mine = (uint64_t)lo | ((uint64_t)hi << 32);
  }
  return mine;
}

// A tile of the rate kernel.
struct RateTile {
  int slot[TILE_BRICKS];
  int entry[TILE_BRICKS];      // its place in the slot list
  int first[TILE_BRICKS];      // list position of the brick's first active cell
  uint64_t act[TILE_BRICKS][8];
  int sums[RATE_THREADS / 32];
  int count, dom, next;
  unsigned long long rbase;
  uint16_t terms[VLSG_MAX_MATERIALS];
  uint16_t list[TILE_LIST];    // brick of the tile << 9 | cell
};

// LocalLaxFriedrichs takes 27 velocities a point, at the normals of the cells of
// its box, and neighbouring points share most of those cells: a round's bricks'
// box normals (the brick and one cell around it, BOX_CELLS each) are computed
// once, in shared memory, for the cells next to an active one, and every point
// reads its 27.  About 10 normals a point instead of 27 (each 7 reads, 6
// divisions, a square root and a reciprocal).  48 KB: 4 bricks for float, 2 for
// double, whose points keep most of a block busy; shared memory would hold three
// blocks per SM (float runs three, double two: rateMinBlocks).
// Rate kernel, one B200: 24 FP32 domains, 0.9M active points, 0.79 -> 0.45 ms; FP64
// trench, 18.5k points, 88 -> 70 us; with reflective walls 215 -> 78 us.
template <class T> constexpr int boxBricks() { return sizeof(T) == 4 ? 4 : 2; }
template <class T> constexpr size_t boxBytes() {
  return (size_t)boxBricks<T>() * 3 * BOX_CELLS * sizeof(T);
}
extern __shared__ __align__(16) unsigned char rateShared[];

template <class T>
__device__ inline void boxTile(const RateArgs<T> &A, RateTile &ts, int m, T gridDelta, T *normals) {
  constexpr int EDGE = BOX_EDGE, ROWS = EDGE * EDGE;
  __shared__ uint16_t rows[boxBricks<T>()][BS * BS]; // active cells of an x-row, widened by one
  const int tid = threadIdx.x;
  for (int e = tid; e < m * BS * BS; e += RATE_THREADS) {
    const unsigned b = (unsigned)(ts.act[e >> 6][(e >> 3) & 7] >> (8 * (e & 7))) & 0xffu;
    rows[e >> 6][e & 63] = (uint16_t)(b | (b << 1) | (b << 2));
  }
  __syncthreads();
  // cells of the box rows tid and tid + RATE_THREADS next to an active cell
  constexpr int PER = (boxBricks<T>() * ROWS + RATE_THREADS - 1) / RATE_THREADS;
  unsigned need[PER];
  int count = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int e = tid + k * RATE_THREADS;
    need[k] = 0u;
    if (e < m * ROWS) {
      const int i = e / ROWS, y = e % ROWS % EDGE, z = e % ROWS / EDGE;
      for (int dz = max(z - 2, 0); dz <= min(z, BS - 1); ++dz)
        for (int dy = max(y - 2, 0); dy <= min(y, BS - 1); ++dy) need[k] |= rows[i][dz * BS + dy];
    }
    count += __popc(need[k]);
  }
  int cells;
  int at = tileScan(ts.sums, count, &cells);
#pragma unroll
  for (int k = 0; k < PER; ++k)
    for (unsigned w = need[k]; w; w &= w - 1)
      ts.list[at++] = (uint16_t)((tid + k * RATE_THREADS) * EDGE + __ffs(w) - 1);
  __syncthreads();
  for (int k = tid; k < cells; k += RATE_THREADS) {
    const int i = ts.list[k] / BOX_CELLS, c = ts.list[k] % BOX_CELLS;
    T normal[3];
    withStencilAt<T, 1>(A, ts.slot[i], c % EDGE - 1, c / EDGE % EDGE - 1, c / ROWS - 1,
                        [&](const auto &S) { boxNormal<T>(S, gridDelta, 0, 0, 0, normal); });
    for (int d = 0; d < 3; ++d) normals[(3 * i + d) * BOX_CELLS + c] = normal[d];
  }
  __syncthreads();
}

// Resident blocks per SM: 3 for float (80 registers), 4 for the float WENO
// kernels (64 registers: a few spilled values, 8% faster than 3 blocks), 2
// for double (the FP64 stencils need 128 registers to stay out of local
// memory).
template <class T, int FAM = FAM_ANY> constexpr int rateMinBlocks() {
  return sizeof(T) == 4 ? (FAM == FAM_WENO ? 4 : 3) : 2;
}
// MODE 0: rates (integrateTime); MODE 1: the global alphas of the
// Lax-Friedrichs schemes (findGlobalAlphas).  TABLE: velocities from the
// host callback's table instead of the device functor.
// BATCH: the batching form (per-domain spacing, velocity and reductions,
// A.slotDom set).
// MINB: resident blocks per SM to compile for (0: rateMinBlocks), the launch
// shapes the batching form's autotuner chooses from.
template <class T, int MODE, bool TABLE = false, int FAM = FAM_ANY, bool BATCH = false, int MINB = 0>
__global__ void __launch_bounds__(RATE_THREADS, MINB ? MINB : rateMinBlocks<T, FAM>())
    kRates(RateArgs<T> A, const vlsg_velocity_desc desc) {
  __shared__ RateTile ts;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int warp = blockIdx.x * (RATE_THREADS / 32) + wid;
  const int n = *A.nSlots;
  const int L = A.L;
  const Buf<T> &top = A.ls[L - 1];
  unsigned long long minBits = ~0ull, alphaMax[3] = {0, 0, 0}, nAct = 0, nBand = 0;
  // StencilLLF: HRLE key and finalAlphas of this thread's last passing call
  unsigned long long lastKey = 0;
  T lastAlpha[3] = {0, 0, 0};
  // batching form: the domain whose partial reductions the registers hold;
  // they go to its RED_* words when the block moves to another domain's bricks
  int dom = -1;
  double delta = A.g.delta;
  const auto flushDomain = [&] {
    minBits = warpMinU64(minBits);
    for (int d = 0; d < 3; ++d) alphaMax[d] = warpMaxU64(alphaMax[d]);
    for (int o = 16; o > 0; o >>= 1) nAct += __shfl_xor_sync(0xffffffffu, nAct, o);
    if (lane == 0) {
      unsigned long long *red = A.domRed + (size_t)RED_WORDS * dom;
      if (MODE == 0 && minBits != ~0ull) atomicMin(red + RED_MIN, minBits);
      for (int d = 0; d < 3; ++d)
        if (alphaMax[d]) atomicMax(red + RED_ALPHA + d, alphaMax[d]);
      if (MODE == 0 && nAct) atomicAdd(red + RED_ACTIVE, nAct);
    }
    minBits = ~0ull, alphaMax[0] = alphaMax[1] = alphaMax[2] = 0, nAct = nBand = 0;
  };
  if (!TABLE && !BATCH && tid < VLSG_MAX_MATERIALS) ts.terms[tid] = velocityTerms<T>(desc, tid);
  const int per = min(TILE_BRICKS, tileEntries(n));
  const int tiles = (n + per - 1) / per;
  // `next`: first list entry of the tile not done yet (a round takes at most
  // tileMost bricks, in the batching form of one domain)
  constexpr int tileMost = FAM == FAM_BOX ? boxBricks<T>() : TILE_BRICKS;
  for (int tile = blockIdx.x, next = tile * per; tile < tiles;) {
    const int end = min((tile + 1) * per, n);
    if (wid == 0) {
      const int e = next + lane;
      const bool in = e < end;
      const int slot = in ? A.slotList[e] : 0;
      const bool go = in && (!A.visit || A.visit[slot]); // else no defined cell
      const unsigned mask = __ballot_sync(0xffffffffu, go);
      const int p = __popc(mask & ((1u << lane) - 1));
      bool over = go && p >= tileMost;
      if constexpr (BATCH) {
        const int d = in ? A.slotDom[slot] : -1;
        const int d0 = __shfl_sync(0xffffffffu, d, mask ? __ffs(mask) - 1 : 0);
        over |= go && d != d0;
        if (lane == 0) ts.dom = d0;
      }
      const unsigned later = __ballot_sync(0xffffffffu, over);
      const int stop = later ? next + __ffs(later) - 1 : end;
      if (e < stop) {
        if (go) {
          ts.slot[p] = slot;
          ts.entry[p] = e;
        } else if (MODE == 0 && in) {
          uint4 *w = reinterpret_cast<uint4 *>(A.act + (size_t)slot * 8);
          for (int k = 0; k < 4; ++k) w[k] = make_uint4(0u, 0u, 0u, 0u);
        }
      }
      if (lane == 0) ts.count = __popc(later ? mask & ((1u << (__ffs(later) - 1)) - 1) : mask), ts.next = stop;
    }
    __syncthreads();
    const int m = ts.count;
    next = ts.next;
    if constexpr (BATCH) {
      if (ts.dom != dom) {
        if (dom >= 0) flushDomain();
        dom = ts.dom;
        delta = A.domDelta[dom];
        if (tid < VLSG_MAX_MATERIALS) ts.terms[tid] = velocityTerms<T>(A.domVel[dom], tid);
      }
    }
    // the bricks' active cells, a warp per brick
    for (int i = wid; i < m; i += RATE_THREADS / 32) {
      const int slot = ts.slot[i];
      const uint64_t own = lane < 8 ? A.def[(size_t)slot * 8 + lane] : 0ull;
      uint64_t a = 0ull;
      if (__any_sync(0xffffffffu, own != 0ull)) a = activePlanes<T>(top.vals, slot);
      int z0 = 0;
      if (A.ownZ) {
        int bx, by, bz;
        brickCoords(A.g, A.m.slotBrick[slot], bx, by, bz);
        z0 = A.g.org[2] + bz * BS;
      }
      if (lane < 8) {
        ts.act[i][lane] = a;
        if (MODE == 0) A.act[(size_t)slot * 8 + lane] = a;
        const bool planeOwned = !A.ownZ || (z0 + lane >= A.ownLo && z0 + lane < A.ownHi);
        if (planeOwned) {
          nAct += __popcll(a);
          nBand += __popcll(own);
        }
      }
    }
    __syncthreads();
    // one thread per plane: the tile's list of active cells
    const int i = tid >> 3, z = tid & 7;
    uint64_t left = i < m ? ts.act[i][z] : 0ull;
    int total;
    int at = tileScan(ts.sums, __popcll(left), &total);
    if (i < m && z == 0) ts.first[i] = at;
    // MODE 0: the tile's entries in the compact rate arrays; a pool that is
    // too small leaves the tile out (the host sees rateNext > rateCap, grows
    // the arrays and runs the pass again)
    if (MODE == 0 && total && tid == 0) {
      const unsigned long long r = atomicAdd(A.rateNext, (unsigned long long)total);
      const bool fits = r + (unsigned long long)total <= A.rateCap;
      if (!fits && A.rateOverflowErr) atomicOr(A.err, A.rateOverflowErr);
      ts.rbase = fits ? r : ~0ull;
    }
    __syncthreads();
    const unsigned long long rbase = MODE == 0 && total ? ts.rbase : 0ull;
    T *boxNormals = nullptr;
    if constexpr (FAM == FAM_BOX) {
      boxNormals = reinterpret_cast<T *>(rateShared);
      if (total) boxTile(A, ts, m, T(delta), boxNormals);
    }
    if (MODE == 0 && rbase != ~0ull && i < m && z == 0) A.rateBase[ts.slot[i]] = rbase + at;
    for (int w0 = 0; w0 < total && rbase != ~0ull; w0 += TILE_LIST) {
      const int size = min(TILE_LIST, total - w0);
      while (left && at < w0 + size) {
        ts.list[at++ - w0] = (uint16_t)((i << 9) | (z << 6) | (__ffsll((long long)left) - 1));
        left &= left - 1;
      }
      __syncthreads();
      for (int kk = tid; kk < size; kk += RATE_THREADS) {
        const int bi = ts.list[kk] >> 9, c = ts.list[kk] & (BV - 1);
        const int slot = ts.slot[bi];
        const int k = w0 + kk - ts.first[bi]; // rank within the brick
        const auto vel = [&] {
          if constexpr (TABLE) {
            const size_t p = (size_t)A.actOff[ts.entry[bi]] + k;
            return TableVel{A.velS, A.velV, p * L * A.velSites, A.velSites, A.alphaTab, p * L * 81,
                            A.velS2, p * L * 162};
          } else if constexpr (BATCH) {
            return FunctorVel{A.domVel[dom], ts.terms};
          } else {
            return FunctorVel{desc, ts.terms};
          }
        }();
        int z0 = 0;
        if (A.ownZ) {
          int bx, by, bz;
          brickCoords(A.g, A.m.slotBrick[slot], bx, by, bz);
          z0 = A.g.org[2] + bz * BS;
        }
        const bool owned = !A.ownZ || (z0 + (c >> 6) >= A.ownLo && z0 + (c >> 6) < A.ownHi);
        withStencil<T>(A, slot, c, [&](const auto &S, T value) {
          if constexpr (MODE == 0) {
            constexpr bool STENCIL = FAM == FAM_STENCIL;
            T alphas[STENCIL ? 4 : 3] = {};
            const double step =
                ratePoint<T, std::decay_t<decltype(S)>, std::decay_t<decltype(vel)>, FAM>(
                    A, vel, S, slot, c, value, alphas, delta, (size_t)(rbase + w0 + kk),
                    FAM == FAM_BOX ? boxNormals + 3 * BOX_CELLS * bi +
                                         ((c >> 6) + 1) * BOX_EDGE * BOX_EDGE +
                                         (((c >> 3) & 7) + 1) * BOX_EDGE + (c & 7) + 1
                                   : nullptr);
            if (!owned) return; // a ghost point: advanced, not counted
            const unsigned long long sb = stepBits(step);
            minBits = sb < minBits ? sb : minBits;
            if constexpr (STENCIL) {
              if (alphas[3] != T(0)) {
                int bx, by, bz;
                brickCoords(A.g, A.m.slotBrick[slot], bx, by, bz);
                const unsigned long long x = A.g.org[0] + bx * BS + (c & 7) + (1 << 20),
                                         y = A.g.org[1] + by * BS + ((c >> 3) & 7) + (1 << 20),
                                         z = A.g.org[2] + bz * BS + (c >> 6) + (1 << 20);
                const unsigned long long key = (z << 42) | (y << 21) | x;
                if (key > lastKey) {
                  lastKey = key;
                  for (int d = 0; d < 3; ++d) lastAlpha[d] = alphas[d];
                }
              }
            } else {
              for (int d = 0; d < 3; ++d) {
                const unsigned long long ab = alphaBits((double)alphas[d]);
                alphaMax[d] = ab > alphaMax[d] ? ab : alphaMax[d];
              }
            }
          } else {
            for (int lower = 0; lower < L; ++lower) {
              const T lv = lower == L - 1 ? value : lsValueAt<T>(A.ls[lower], slot, c);
              if ((double)lv <= (double)value + 1e-4) {
                T normal[3];
                T normalModulus = 0.;
                for (int d = 0; d < 3; ++d) {
                  const T phiPos = S.axis(d, 1);
                  const T phiNeg = S.axis(d, -1);
                  normal[d] = phiPos - phiNeg;
                  normalModulus += normal[d] * normal[d];
                }
                normalModulus = T(1.) / sqrt(normalModulus);
                for (int d = 0; d < 3; ++d) normal[d] *= normalModulus;
                T scaVel, vecVel[3];
                vel.get(lower, normal, 0, scaVel, vecVel);
                if (owned)
                  for (int d = 0; d < 3; ++d) {
                    const unsigned long long ab =
                        alphaBits((double)fabs((scaVel + vecVel[d]) * normal[d]));
                    alphaMax[d] = ab > alphaMax[d] ? ab : alphaMax[d];
                  }
                break;
              }
            }
          }
        });
      }
      __syncthreads();
    }
    __syncthreads();
    if (next >= end) tile += gridDim.x, next = tile * per;
  }
  if constexpr (FAM == FAM_STENCIL && MODE == 0) {
    const unsigned long long best = warpMaxU64(lastKey);
    const unsigned owner = __ballot_sync(0xffffffffu, best != 0ull && lastKey == best);
    if (best == 0ull ? lane == 0 : (owner >> lane) & 1u) {
      A.sllfKey[warp] = best;
      for (int d = 0; d < 3; ++d) A.sllfAlpha[3 * warp + d] = (double)lastAlpha[d];
    }
  }
  if constexpr (BATCH) {
    if (dom >= 0) flushDomain();
    return;
  }
  minBits = warpMinU64(minBits);
  for (int d = 0; d < 3; ++d) alphaMax[d] = warpMaxU64(alphaMax[d]);
  for (int o = 16; o > 0; o >>= 1) {
    nAct += __shfl_xor_sync(0xffffffffu, nAct, o);
    nBand += __shfl_xor_sync(0xffffffffu, nBand, o);
  }
  if (lane == 0) {
    if (MODE == 0 && minBits != ~0ull) atomicMax(A.minStep, ~minBits);
    if (A.alphaMax)
      for (int d = 0; d < 3; ++d)
        if (alphaMax[d]) atomicMax(&A.alphaMax[d], alphaMax[d]);
    if (MODE == 0 && A.counts) {
      if (nAct) atomicAdd(&A.counts[0], nAct);
      if (nBand) atomicAdd(&A.counts[1], nBand);
    }
  }
}

// StencilLocalLaxFriedrichs time-step alphas: the finalAlphas of the warp
// entry with the largest HRLE key (the last passing call in HRLE order) go to
// alphaOut[0..2] as double bits; nothing is written when no call passed.
__global__ void __launch_bounds__(1024)
    kSllfPick(const unsigned long long *key, const double *alpha, int n,
              unsigned long long *alphaOut) {
  __shared__ unsigned long long sk[32];
  __shared__ int si[32];
  unsigned long long best = 0;
  int bi = -1;
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    if (key[i] > best) best = key[i], bi = i;
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long k2 = __shfl_xor_sync(0xffffffffu, best, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
    if (k2 > best) best = k2, bi = i2;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sk[wid] = best, si[wid] = bi;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
      if (sk[w] > best) best = sk[w], bi = si[w];
    if (best != 0ull && bi >= 0)
      for (int d = 0; d < 3; ++d) alphaOut[d] = (unsigned long long)__double_as_longlong(alpha[3 * bi + d]);
  }
}

// Value update of one active point (updateLevelSet, lsAdvect.hpp:725-777): the
// stop chain walked with the time step; entry j of the point's rates is at
// j * rateCap + r.
template <class T> struct UpdateArgs {
  const T *rateV, *rateStop;
  const uint8_t *rateLen;
  const unsigned long long *rateBase;
  size_t rateCap;
  int L;
  int *err;
  float *lo;      // compensation terms (FP32 buffers that carry them), or null
  T *pvel, *pdiss; // setSaveAdvectionVelocities, else null: the point's last leg
                   // rate (time x velocity) and the dissipation of the chain
                   // entry it ended on, lsAdvect.hpp:764-767
  const T *rateD;
};
template <class T>
__device__ inline T updatedValue(const UpdateArgs<T> &A, size_t r, size_t q, T old, double time) {
  int len = A.rateLen[r];
  if (len < 1 || len > A.L) {
    atomicOr(A.err, 2);
    len = 1;
  }
  int j = 0;
  if constexpr (sizeof(T) == 4) {
    if (A.lo) {
      // the value is hi + lo: the walk runs in double, the result is split again
      double value = withLo((double)old, A.lo[q]);
      double velocity = A.rateV[r];
      double rate = time * velocity;
      while (fabs((double)A.rateStop[(size_t)j * A.rateCap + r] - value) < fabs(rate)) {
        const double stop = A.rateStop[(size_t)j * A.rateCap + r];
        time -= fabs((stop - value) / velocity);
        value = stop;
        ++j;
        if (j >= len) {
          atomicOr(A.err, 2);
          break;
        }
        velocity = A.rateV[(size_t)j * A.rateCap + r];
        rate = time * velocity;
      }
      value -= rate;
      const float hi = (float)value;
      A.lo[q] = (float)(value - (double)hi);
      if (A.pvel) {
        const int jj = j < len ? j : len - 1; // j == len only after a chain overrun
        A.pvel[q] = T(rate), A.pdiss[q] = A.rateD[(size_t)jj * A.rateCap + r];
      }
      return hi;
    }
  }
  T value = old;
  T velocity = A.rateV[r];
  T rate = T(time * velocity);
  while (fabs(A.rateStop[(size_t)j * A.rateCap + r] - value) < fabs(rate)) {
    const T stop = A.rateStop[(size_t)j * A.rateCap + r];
    time -= fabs((stop - value) / velocity);
    value = stop;
    ++j;
    if (j >= len) {
      atomicOr(A.err, 2);
      break;
    }
    velocity = A.rateV[(size_t)j * A.rateCap + r];
    rate = T(time * velocity);
  }
  value -= rate;
  if (A.pvel) {
    const int jj = j < len ? j : len - 1; // j == len only after a chain overrun
    A.pvel[q] = rate, A.pdiss[q] = A.rateD[(size_t)jj * A.rateCap + r];
  }
  return value;
}

// updateLevelSet: every active point takes its new value and every other
// defined cell becomes undefined with its sign (Reduce(1), lsReduce.hpp:
// 285-296), in place; afterwards `act` are the level set's masks.  rebuildLS
// then runs as an ordinary band pass (kFrontierPass).
//
// Tiles of bricks as in kRates: a warp streams a brick's defined cells that
// are not active, four groups of 32 in flight; the tile's active cells are one
// list, a thread each (a point's rate entry is the brick's first plus the
// active cells before it), so that the loads of many chain walks overlap.
// FP32 sphere of 16.8M band points, update + rebuild of a stage: 0.23 + 1.06 ms
// before (the rebuild did the reduction and fetched an active word next to
// every neighbour value), 0.31 + 0.52 ms now; walking the chains group by group
// of the stream, one after another in flight, took 0.93 + 0.52 ms.  Resident
// blocks per SM: 6 for float (40 registers), 4 for double.
template <class T> constexpr int updateMinBlocks() { return sizeof(T) == 4 ? 6 : 4; }
template <class T>
__global__ void __launch_bounds__(RATE_THREADS, updateMinBlocks<T>())
    kUpdate(const int *slotList, const int *nSlots, const uint64_t *act, const uint64_t *def,
            const uint8_t *visitIn, T *vals, UpdateArgs<T> A, double dt, const int *slotDom,
            const double *domDt) {
  __shared__ RateTile ts;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int n = *nSlots;
  const int per = min(TILE_BRICKS, tileEntries(n));
  const int tiles = (n + per - 1) / per;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    if (wid == 0) {
      const int e = tile * per + lane;
      const bool in = lane < per && e < n;
      const int slot = in ? slotList[e] : 0;
      const bool go = in && (!visitIn || visitIn[slot]);
      const unsigned mask = __ballot_sync(0xffffffffu, go);
      if (go) ts.slot[__popc(mask & ((1u << lane) - 1))] = slot;
      if (lane == 0) ts.count = __popc(mask);
    }
    __syncthreads();
    const int m = ts.count;
    // one thread per plane: the list of active cells
    const int i = tid >> 3, z = tid & 7;
    uint64_t left = i < m ? act[(size_t)ts.slot[i] * 8 + z] : 0ull;
    int total;
    int at = tileScan(ts.sums, __popcll(left), &total);
    if (i < m && z == 0) ts.first[i] = at;
    // a warp per brick: the other defined cells
    for (int b = wid; b < m; b += RATE_THREADS / 32) {
      const size_t slot = ts.slot[b];
      const unsigned mine = lane < 16 ? reinterpret_cast<const unsigned *>(def)[slot * 16 + lane] &
                                            ~reinterpret_cast<const unsigned *>(act)[slot * 16 + lane]
                                      : 0u;
      if (!__any_sync(0xffffffffu, mine != 0u)) continue;
      T *p = vals + slot * BV + lane;
#pragma unroll
      for (int g = 0; g < 16; g += 4) {
        T v[4];
        bool on[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          on[k] = (__shfl_sync(0xffffffffu, mine, g + k) >> lane) & 1u;
          v[k] = on[k] ? p[(g + k) * 32] : T(0);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (on[k]) p[(g + k) * 32] = sentinel<T>(v[k] < 0);
      }
    }
    for (int w0 = 0; w0 < total; w0 += TILE_LIST) {
      const int size = min(TILE_LIST, total - w0);
      while (left && at < w0 + size) {
        ts.list[at++ - w0] = (uint16_t)((i << 9) | (z << 6) | (__ffsll((long long)left) - 1));
        left &= left - 1;
      }
      __syncthreads();
      for (int k = tid; k < size; k += RATE_THREADS) {
        const int b = ts.list[k] >> 9, c = ts.list[k] & (BV - 1);
        const int slot = ts.slot[b];
        const size_t q = (size_t)slot * BV + c;
        const size_t r = (size_t)A.rateBase[slot] + (w0 + k - ts.first[b]);
        if (r >= A.rateCap) { // the rate pass left this brick out (storage too small)
          atomicOr(A.err, 1024);
          continue;
        }
        // batching form: the time step of the slot's domain
        vals[q] = updatedValue(A, r, q, vals[q], domDt ? domDt[slotDom[slot]] : dt);
      }
      __syncthreads();
    }
    __syncthreads();
  }
}

} // namespace
} // namespace vlsg
