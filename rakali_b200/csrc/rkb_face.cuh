// Face-level numerics of the structured barotropic flux.
//
// Templates on the real type T (double in the production step and the FP64
// adjoint, float in the FP32 adjoint); constants enter as T(c).
//
// One call evaluates one cell face: Audusse hydrostatic reconstruction of the
// two side states, then the HLL or HLLC Riemann flux.  The reference
// (rki_kernel_flux.F90:104-378, flux_cell) evaluates every interior face
// twice, once from each neighbour, and the two evaluations are bit-identical;
// the B200 kernels evaluate each face once and share it through shared memory.
#pragma once

#include <type_traits>

#include "rkb_common.cuh"
#include "rkb_rnmath.cuh"

namespace rkb {

// Outputs of one face.  wbR is the right-side well-balanced term
// h_hyd^2 - h_pre^2 (the neighbour to the right adds it first); hL2 and pL2
// are the left side's h_hyd^2 and h_pre^2, subtracted and added in that order
// by the neighbour to the left (rki_kernel_flux.F90:361-369).
template <typename T>
struct FaceOutT {
  T fh, fqx, fqy;
  T wbR, hL2, pL2;
};
using FaceOut = FaceOutT<double>;

template <typename T>
__host__ __device__ __forceinline__ void velocity(T h, T qx, T qy, T& u, T& v) {
  if (h > T(kDry)) {
    u = qx / h;
    v = qy / h;
  } else {
    u = T(0);
    v = T(0);
  }
}

// HLL / HLLC in direction DIR (0: x, normal momentum qx; 1: y, normal qy).
// hll_flux_x/y rki_kernel_flux.F90:410-582, hllc_flux_x/y :584-783.
template <int DIR, bool HLLC, typename T>
__host__ __device__ __forceinline__ void riemann(T hl, T qxl, T qyl, T hr, T qxr, T qyr, T& fh,
                                                 T& fqx, T& fqy) {
  T ul, vl, ur, vr;
  velocity(hl, qxl, qyl, ul, vl);
  velocity(hr, qxr, qyr, ur, vr);
  const T al = sqrt(T(kG) * pos(hl));
  const T ar = sqrt(T(kG) * pos(hr));
  const T nl = DIR == 0 ? ul : vl;
  const T nr = DIR == 0 ? ur : vr;
  T sl, sr;
  if (hr <= T(kDry)) {
    sl = nl - al;
    sr = nl + T(2) * al;
  } else if (hl <= T(kDry)) {
    sl = nr - T(2) * ar;
    sr = nr + ar;
  } else {
    sl = dmin(nl - al, nr - ar);
    sr = dmax(nl + al, nr + ar);
  }
  T lh, lx, ly, rh, rx, ry;
  if (DIR == 0) {
    lh = qxl;
    lx = qxl * ul + T(kHalfG) * hl * hl;
    ly = qxl * vl;
    rh = qxr;
    rx = qxr * ur + T(kHalfG) * hr * hr;
    ry = qxr * vr;
  } else {
    lh = qyl;
    lx = qxl * vl;
    ly = qyl * vl + T(kHalfG) * hl * hl;
    rh = qyr;
    rx = qxr * vr;
    ry = qyr * vr + T(kHalfG) * hr * hr;
  }
  if (sl >= T(0)) {
    fh = lh; fqx = lx; fqy = ly;
    return;
  }
  if (sr <= T(0)) {
    fh = rh; fqx = rx; fqy = ry;
    return;
  }
  const T inv = T(1) / (sr - sl);
  const T slsr = sl * sr;
  fh = (sr * lh - sl * rh + slsr * (hr - hl)) * inv;
  if (DIR == 0) {
    fqx = (sr * lx - sl * rx + slsr * (qxr - qxl)) * inv;
    if (!HLLC) {
      fqy = (sr * ly - sl * ry + slsr * (qyr - qyl)) * inv;
    } else {
      const T den = hr * (ur - sr) - hl * (ul - sl);
      T ss;
      if (fabs(den) > T(kDry))
        ss = (sl * hr * (ur - sr) - sr * hl * (ul - sl)) / den;
      else
        ss = T(0.5) * (ul + ur);
      fqy = ss >= T(0) ? fh * vl : fh * vr;
    }
  } else {
    fqy = (sr * ly - sl * ry + slsr * (qyr - qyl)) * inv;
    if (!HLLC) {
      fqx = (sr * lx - sl * rx + slsr * (qxr - qxl)) * inv;
    } else {
      const T den = hr * (vr - sr) - hl * (vl - sl);
      T ss;
      if (fabs(den) > T(kDry))
        ss = (sl * hr * (vr - sr) - sr * hl * (vl - sl)) / den;
      else
        ss = T(0.5) * (vl + vr);
      fqx = ss >= T(0) ? fh * ul : fh * ur;
    }
  }
}

// One face from the reconstructed side values (eta, hu, hv) and the beds.
// The Audusse step follows rki_kernel_flux.F90:186-224.
template <int DIR, bool HLLC, typename T>
__host__ __device__ __forceinline__ void face_flux(T eL, T qxL, T qyL, T bL, T eR, T qxR, T qyR,
                                                   T bR, FaceOutT<T>& o) {
  const T hL = pos(eL - bL);
  const T hR = pos(eR - bR);
  const T bmax = dmax(bL, bR);
  const T hyl = pos(hL + bL - bmax);
  const T hyr = pos(hR + bR - bmax);
  T ul, vl, ur, vr;
  velocity(hL, qxL, qyL, ul, vl);
  velocity(hR, qxR, qyR, ur, vr);
  riemann<DIR, HLLC>(hyl, hyl * ul, hyl * vl, hyr, hyr * ur, hyr * vr, o.fh, o.fqx, o.fqy);
  o.wbR = hyr * hyr - hR * hR;
  o.hL2 = hyl * hyl;
  o.pL2 = hL * hL;
}

// Limited slope of one cell along one direction (rki_kernel_flux.F90:159-181):
// zero near wet/dry fronts, else minmod of the one-sided differences.
template <typename T>
__host__ __device__ __forceinline__ void cell_slope(T hm, T hc, T hp, T em, T ec, T ep, T um, T uc,
                                                    T up, T vm, T vc, T vp, T& se, T& su, T& sv) {
  if (hc < T(kThin) || hm < T(kDry) || hp < T(kDry)) {
    se = T(0); su = T(0); sv = T(0);
  } else {
    se = minmod(ec - em, ep - ec);
    su = minmod(uc - um, up - uc);
    sv = minmod(vc - vm, vp - vc);
  }
}

// ---- faces between two wet cells, FP64 --------------------------------------
//
// face_flux for the ordinary face: both reconstructed depths and both
// hydrostatic depths above the dry threshold, every operand of moderate size
// (moderate() below).  The same expressions in the same order with the
// quotients of rkb_rnmath.cuh, hence the same bits, without their range tests:
// the two velocities of a side share one reciprocal of its depth, and the
// quotients (h_hyd u) / h_hyd, which only undo a product, take a remainder step
// each.  The HLLC contact speed enters through its sign alone, which is that of
// numerator and denominator together.  Returns false for any other face (`o`
// then holds nothing).

// Tile values for which every operand of the faces and of the divergence
// stays within the range rkb_rnmath.cuh asks for: depth and momenta zero or
// above 2^-250, nothing above 2^40 in sum (products of two momenta and their
// differences then stay above 2^-850, remainders above the subnormals).
__device__ __forceinline__ bool moderate(double h, double u, double v, double b) {
  constexpr double lo = 0x1p-250;
  return fabs(h) + fabs(u) + fabs(v) + fabs(b) < 0x1p40 && (h == 0.0 || fabs(h) >= lo) &&
         (u == 0.0 || fabs(u) >= lo) && (v == 0.0 || fabs(v) >= lo);
}

// The same for the inputs of one face.
__device__ __forceinline__ bool moderate_face(double eL, double qxL, double qyL, double bL,
                                              double eR, double qxR, double qyR, double bR) {
  constexpr double lo = 0x1p-300;
  return fabs(eL) + fabs(qxL) + fabs(qyL) + fabs(bL) + fabs(eR) + fabs(qxR) + fabs(qyR) + fabs(bR) <
             0x1p42 &&
         (qxL == 0.0 || fabs(qxL) >= lo) && (qyL == 0.0 || fabs(qyL) >= lo) &&
         (qxR == 0.0 || fabs(qxR) >= lo) && (qyR == 0.0 || fabs(qyR) >= lo);
}

template <int DIR, bool HLLC>
__device__ __forceinline__ bool face_flux_wet(double eL, double qxL, double qyL, double bL,
                                              double eR, double qxR, double qyR, double bR,
                                              FaceOut& o) {
  const double hL = eL - bL, hR = eR - bR;
  const double bmax = dmax(bL, bR);
  const double hl = hL + bL - bmax, hr = hR + bR - bmax;
  // integer tests beside the FP64 pipe: all four depths clear of the threshold
  // (values next to it say no), none with a significand of all ones
  // (last_bits_set)
  const int high = min(min(__double2hiint(hL), __double2hiint(hR)),
                       min(__double2hiint(hl), __double2hiint(hr)));
  const unsigned low = max(max((unsigned)__double2loint(hL), (unsigned)__double2loint(hR)),
                           max((unsigned)__double2loint(hl), (unsigned)__double2loint(hr)));
  if (high <= 0x3eb0c6f7 || low == 0xffffffffu) return false;  // the high word of 1e-6
  double ul, vl, ur, vr, qxl, qyl, qxr, qyr;
  {
    const double y = rcp_near(hL);
    ul = quot_by(qxL, hL, y);
    vl = quot_by(qyL, hL, y);
  }
  {
    const double y = rcp_near(hR);
    ur = quot_by(qxR, hR, y);
    vr = quot_by(qyR, hR, y);
  }
  qxl = hl * ul;
  qyl = hl * vl;
  qxr = hr * ur;
  qyr = hr * vr;
  {
    const double y = rcp_near(hl);
    ul = requot_by(qxl, hl, y, ul);
    vl = requot_by(qyl, hl, y, vl);
  }
  {
    const double y = rcp_near(hr);
    ur = requot_by(qxr, hr, y, ur);
    vr = requot_by(qyr, hr, y, vr);
  }
  const double al = sqrt_rn(kG * hl), ar = sqrt_rn(kG * hr);
  const double nl = DIR == 0 ? ul : vl, nr = DIR == 0 ? ur : vr;
  const double sl = dmin(nl - al, nr - ar), sr = dmax(nl + al, nr + ar);
  double lh, lx, ly, rh, rx, ry;
  if (DIR == 0) {
    lh = qxl;
    lx = qxl * ul + kHalfG * hl * hl;
    ly = qxl * vl;
    rh = qxr;
    rx = qxr * ur + kHalfG * hr * hr;
    ry = qxr * vr;
  } else {
    lh = qyl;
    lx = qxl * vl;
    ly = qyl * vl + kHalfG * hl * hl;
    rh = qyr;
    rx = qxr * vr;
    ry = qyr * vr + kHalfG * hr * hr;
  }
  const double w = sr - sl;
  const double inv = rcp_rn(w);
  const double slsr = sl * sr;
  o.fh = (sr * lh - sl * rh + slsr * (hr - hl)) * inv;
  if (DIR == 0 || !HLLC) o.fqx = (sr * lx - sl * rx + slsr * (qxr - qxl)) * inv;
  if (DIR == 1 || !HLLC) o.fqy = (sr * ly - sl * ry + slsr * (qyr - qyl)) * inv;
  if (HLLC) {
    const double cl = nl - sl, cr = nr - sr;
    const double den = hr * cr - hl * cl;
    const double num = sl * hr * cr - sr * hl * cl;
    const bool left = fabs(den) > kDry ? (num == 0.0 || (num < 0.0) == (den < 0.0)) : nl + nr >= 0.0;
    if (DIR == 0)
      o.fqy = o.fh * (left ? vl : vr);
    else
      o.fqx = o.fh * (left ? ul : ur);
  }
  if (!(sl < 0.0 && sr > 0.0 && !last_bits_set(w))) {
    if (sl < 0.0 && sr > 0.0) return false;
    const bool left = sl >= 0.0;  // supercritical
    o.fh = left ? lh : rh;
    o.fqx = left ? lx : rx;
    o.fqy = left ? ly : ry;
  }
  o.hL2 = hl * hl;
  o.pL2 = hL * hL;
  o.wbR = hr * hr - hR * hR;
  return true;
}

// ---- faces of a shared-memory tile, FP64 -------------------------------------

// One face of a tile by the general functions, slopes included: faces next to
// dry or thin cells, and every face of a tile with extreme values.  q: the
// cell on the left (below), d: the index step to the one on the right
// (above); the four tile arrays are `nt` apart, the six outputs `n` apart.
template <int DIR, bool HLLC>
__device__ __noinline__ void face_general(const double* th, int nt, int q, int d, double* f, int n) {
  const double *tu = th + nt, *tv = tu + nt, *tb = tv + nt;
  const double em = th[q - d] + tb[q - d], eL = th[q] + tb[q], eR = th[q + d] + tb[q + d],
               ep = th[q + 2 * d] + tb[q + 2 * d];
  double sLe, sLu, sLv, sRe, sRu, sRv;
  cell_slope(th[q - d], th[q], th[q + d], em, eL, eR, tu[q - d], tu[q], tu[q + d], tv[q - d], tv[q],
             tv[q + d], sLe, sLu, sLv);
  cell_slope(th[q], th[q + d], th[q + 2 * d], eL, eR, ep, tu[q], tu[q + d], tu[q + 2 * d], tv[q],
             tv[q + d], tv[q + 2 * d], sRe, sRu, sRv);
  FaceOut o;
  face_flux<DIR, HLLC>(eL + 0.5 * sLe, tu[q] + 0.5 * sLu, tv[q] + 0.5 * sLv, tb[q],
                       eR - 0.5 * sRe, tu[q + d] - 0.5 * sRu, tv[q + d] - 0.5 * sRv, tb[q + d], o);
  f[0] = o.fh;
  f[n] = o.fqx;
  f[2 * n] = o.fqy;
  f[3 * n] = o.wbR;
  f[4 * n] = o.hL2;
  f[5 * n] = o.pL2;
}

// Value x + side * minmod(a, b) / 2 of one side of a face (rki_kernel_flux.F90:
// 159-181, :380-393) for moderate() values: a b <= 0 is a difference of signs
// or a zero, and halving is exact, so the sum rounds once and is one FMA.  The
// FP64 pipe binds the stage: the test runs beside it, on the high words
// (differences of moderate values are zero or far above the subnormals).
// ZEROS: x may be -0 (a momentum at rest), and the half-slope that is added or
// subtracted then has to be +0.  A surface h + b of a wet cell is never -0, and
// neither the factor's nor the smaller difference's sign matters beside it.
template <bool ZEROS>
__device__ __forceinline__ double limited(double x, double a, double b, double side) {
  const double m = fabs(a) < fabs(b) ? a : b;
  const int signs = __double2hiint(a) ^ __double2hiint(b);
  if (!ZEROS) return __fma_rn(signs >= 0 ? 0.5 * side : 0.0, m, x);
  const int same = (signs & (int)0x80000000) | (__double2hiint(m) & 0x7fffffff);
  return __fma_rn(0.5 * side, same > 0 ? m : 0.0, x);
}

// Above a positive threshold for certain (values next to it may say no);
// an integer comparison.
__device__ __forceinline__ bool clear_of(int hi, double threshold) {
  return hi > __double2hiint(threshold);
}

// The same face in the ordinary case: every cell of its stencil wet and thick
// enough that no slope is gated off, values of moderate size (`mod`, a
// property of the tile).
template <int DIR, bool HLLC>
__device__ __forceinline__ void face_of_tile(const double* th, int nt, int q, int d, double* f,
                                             int n, bool mod) {
  const double *tu = th + nt, *tv = tu + nt, *tb = tv + nt;
  const double hm = th[q - d], hL = th[q], hR = th[q + d], hp = th[q + 2 * d];
  if (mod && clear_of(min(__double2hiint(hL), __double2hiint(hR)), kThin) &&
      clear_of(min(__double2hiint(hm), __double2hiint(hp)), kDry)) {
    const double bL = tb[q], bR = tb[q + d];
    // reconstructed value of both sides of the face
    auto sides = [](auto zeros, double m, double l, double r, double p, double& vl, double& vr) {
      const double a = l - m, b = r - l, c = p - r;
      vl = limited<decltype(zeros)::value>(l, a, b, 1.0);
      vr = limited<decltype(zeros)::value>(r, b, c, -1.0);
    };
    const std::false_type surface;
    const std::true_type momentum;
    double eL, uL, vL, eR, uR, vR;
    sides(surface, hm + tb[q - d], hL + bL, hR + bR, hp + tb[q + 2 * d], eL, eR);
    sides(momentum, tu[q - d], tu[q], tu[q + d], tu[q + 2 * d], uL, uR);
    sides(momentum, tv[q - d], tv[q], tv[q + d], tv[q + 2 * d], vL, vR);
    FaceOut o;
    if (face_flux_wet<DIR, HLLC>(eL, uL, vL, bL, eR, uR, vR, bR, o)) {
      f[0] = o.fh;
      f[n] = o.fqx;
      f[2 * n] = o.fqy;
      f[3 * n] = o.wbR;
      f[4 * n] = o.hL2;
      f[5 * n] = o.pL2;
      return;
    }
  }
  face_general<DIR, HLLC>(th, nt, q, d, f, n);
}

}  // namespace rkb
