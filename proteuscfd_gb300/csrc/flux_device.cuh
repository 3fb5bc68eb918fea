// Device-side equation-set math for the ideal-gas compressible path
// (CompressibleEqnSet<T>, ucs/compressible.tcc), templated on the scalar type:
// S = double is the reference precision, S = dfl runs the same algebra in
// double-float on the FP32 pipes (dfloat.cuh).  Operation order follows the
// reference; divisions by the same quantity are replaced by one reciprocal
// and multiplications, because division and square root are the costliest
// operations on sm_103a.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "dfloat.cuh"
#include "seeded.cuh"

namespace pcfd {

constexpr int NEQN = 5;
constexpr int NVARS = 10;   // rho, rho u, rho v, rho w, rho E | T, P, u, v, w
constexpr int NTERMS = 9;   // gradient terms: 0..5 and 7..9 of q (GetGradientsLocation)

template <class S>
__device__ __forceinline__ S smax(S a, S b) { return (a > b) ? a : b; }

// The generic templates' reciprocal, quotient and root: FP64 from FP32 seeds,
// rounded as the operators round (recip, quot and root are within 2^-10 ulp
// of correct rounding), double-float and FP32 the operators.
__device__ __forceinline__ double inv_s(double x) { return recip(x); }
__device__ __forceinline__ dfl inv_s(dfl x) { return Sc<dfl>::c(1.0) / x; }
__device__ __forceinline__ double div_s(double a, double b) { return quot(a, b); }
__device__ __forceinline__ dfl div_s(dfl a, dfl b) { return a / b; }
__device__ __forceinline__ float div_s(float a, float b) { return a / b; }
__device__ __forceinline__ double sqrt_s(double x) { return root(x); }
__device__ __forceinline__ dfl sqrt_s(dfl x) { return sqrt(x); }
__device__ __forceinline__ float sqrt_s(float x) { return sqrt(x); }
// FP32 estimate (relative error below 2^-22 in FP32's normal range)
__device__ __forceinline__ float est_s(double x) { return est_f32(x); }
__device__ __forceinline__ float est_s(dfl x) { return x.hi; }

// Harten-Hyman entropy fix of one eigenvalue (ucs/compressible.tcc:148-185)
template <class S>
__device__ __forceinline__ S entropy_fix(S eig, S eigL, S eigR) {
  S eps = smax(eig - eigL, eigR - eig);
  eps = smax(Sc<S>::c(0.0), eps);
  S a = fabs(eig);
  if (a < eps) a = halve(div_s(eig * eig, eps) + eps);
  return a;
}

// Primitive quantities of one side of a Roe flux (the per-state part of
// RoeVariables, Eigensystem and Flux): the reciprocal density, velocity,
// pressure, total enthalpy, normal velocity, mass flux rt = rho theta and the
// momentum parts of the physical flux.  A finite-difference Jacobian that
// perturbs one side reuses the other side's record, and the reciprocal density
// of its own where the perturbation leaves the density.
template <class S>
struct RoeSide {
  S r, ir, u, v, w, E, P, h, th, rt, f1, f2, f3;
};
// the part of the Roe average that depends on the densities alone
template <class S>
struct RoePair {
  S rho, sigma;
};

template <class S>
__device__ __forceinline__ RoeSide<S> roe_side_ir(const S* Q, const S ir, const S nx, const S ny, const S nz,
                                                  const S gm1) {
  RoeSide<S> o;
  o.r = Q[0];
  o.ir = ir;
  o.u = Q[1] * o.ir;
  o.v = Q[2] * o.ir;
  o.w = Q[3] * o.ir;
  o.E = Q[4];
  o.P = gm1 * (o.E - halve(o.r) * (o.u * o.u + o.v * o.v + o.w * o.w));
  o.h = (o.E + o.P) * o.ir;
  o.th = o.u * nx + o.v * ny + o.w * nz;
  o.rt = o.r * o.th;
  o.f1 = o.u * o.rt + o.P * nx;
  o.f2 = o.v * o.rt + o.P * ny;
  o.f3 = o.w * o.rt + o.P * nz;
  return o;
}
template <class S>
__device__ __forceinline__ RoeSide<S> roe_side(const S* Q, const S nx, const S ny, const S nz, const S gm1) {
  return roe_side_ir(Q, inv_s(Q[0]), nx, ny, nz, gm1);
}
template <class S>
__device__ __forceinline__ RoePair<S> roe_pair(const S rL, const S rR) {
  RoePair<S> p;
  p.rho = sqrt_s(rL * rR);
  p.sigma = div_s(p.rho, rL + p.rho);
  return p;
}

enum class FuseEnergy { left, right, none };

template <FuseEnergy FUSE>
__device__ __forceinline__ int roe_core64(const RoeSide<double>& L, const RoeSide<double>& R,
                                          const RoePair<double>& pr, const double* QL, const double* QR,
                                          const double nx, const double ny, const double nz, const double area,
                                          const double gamma, const double gm1, const double igamma, double* flux);

// FUSE: which of the energy flux's two products is the fused one in FP64.  The
// residual fuses the left side's; in the finite-difference Jacobian the side a
// column perturbs is the fused one and the base flux rounds both products, the
// roundings its differences have always had.
template <FuseEnergy FUSE = FuseEnergy::left, class S>
__device__ __forceinline__ int roe_core(const RoeSide<S>& L, const RoeSide<S>& R, const RoePair<S>& pr, const S* QL,
                                        const S* QR, const S nx, const S ny, const S nz, const S area, const S gamma,
                                        const S gm1, const S igamma, S* flux);

// Roe flux with the reference's eigensystem: RoeVariables (:533),
// Eigensystem (:580), entropy fix, |A| dQ = T |L| Tinv dQ (evaluated in
// projector form, in roe_core), and 0.5 area (F_L + F_R - |A| dQ)
// (RoeFlux, :93).  (nx, ny, nz, area) is the edge's unit normal and area;
// static grid (vdotn = 0).
// Returns a mask of non-physical states in the sense of BadExtrapolation
// (ucs/compressible.tcc:1056: p < 1e-10, rho < 0 or rho E < 1e-10):
// bit 0 = left state, bit 1 = right state, bit 2 = Roe-averaged state.  The
// limiter's pressure clip (ucs/limiters.tcc:737) applies exactly these
// three tests to the same extrapolated states.
template <class S>
__device__ __forceinline__ int roe_flux(const S* QL, const S* QR, const S nx, const S ny, const S nz, const S area,
                                        const S gamma, const S gm1, const S igamma, const S igm1, S* flux) {
  return roe_core(roe_side(QL, nx, ny, nz, gm1), roe_side(QR, nx, ny, nz, gm1), roe_pair(QL[0], QR[0]), QL, QR, nx,
                  ny, nz, area, gamma, gm1, igamma, flux);
}

// FP32 test that the Harten-Hyman fix cannot apply to the acoustic
// eigenvalues theta +- c: |eig| exceeds the larger of its differences from
// the two sides' values, each at most |dtheta| + |dc| over the pair; the
// margin covers the estimates' errors (2^-20 of the speeds summed)
template <class S>
__device__ __forceinline__ bool acoustics_clear(S theta, S c, S thL, S PL, S irL, S thR, S PR, S irR, S gamma) {
  const float fg = est_s(gamma);
  const float thf = est_s(theta), cf = est_s(c), thl = est_s(thL), thr = est_s(thR);
  const float cl = sqrt_f32(fg * est_s(PL) * est_s(irL)), cr = sqrt_f32(fg * est_s(PR) * est_s(irR));
  const float jump = fmaxf(fabsf(thf - thl), fabsf(thr - thf)) + fmaxf(fabsf(cf - cl), fabsf(cr - cf)) +
                     1.0e-5f * (fabsf(thl) + fabsf(thr) + fabsf(thf) + cl + cr + cf);
  return fabsf(thf + cf) > jump && fabsf(thf - cf) > jump;
}

template <FuseEnergy FUSE, class S>
__device__ __forceinline__ int roe_core(const RoeSide<S>& L, const RoeSide<S>& R, const RoePair<S>& pr, const S* QL,
                                        const S* QR, const S nx, const S ny, const S nz, const S area, const S gamma,
                                        const S gm1, const S igamma, S* flux) {
  if constexpr (std::is_same<S, double>::value)
    return roe_core64<FUSE>(L, R, pr, QL, QR, nx, ny, nz, area, gamma, gm1, igamma, flux);
  const S rL = L.r, uL = L.u, vL = L.v, wL = L.w, EL = L.E, PL = L.P, hL = L.h;
  const S rR = R.r, uR = R.u, vR = R.v, wR = R.w, ER = R.E, PR = R.P, hR = R.h;

  // Roe-averaged state
  const S rho = pr.rho, sigma = pr.sigma;
  const S u = uL + sigma * (uR - uL);
  const S v = vL + sigma * (vR - vL);
  const S w = wL + sigma * (wR - wL);
  const S h = hL + sigma * (hR - hL);
  S v2h = halve(u * u + v * v + w * w);
  const S rE = rho * igamma * (h + gm1 * v2h);
  const S P = gm1 * (rE - rho * v2h);
  const S c2 = gm1 * (h - v2h);  // = gamma P / rho with P and rE above
  const S c = sqrt_s(c2);
  const S ic2 = inv_s(c2);
  const S thetaf = u * nx + v * ny + w * nz;

  // entropy-fixed |eigenvalues|; the sides' acoustic speeds are formed only
  // where the fix of an acoustic one may apply
  const S thetaL = L.th, thetaR = R.th;
  const S l0 = entropy_fix(thetaf, thetaL, thetaR);
  S l3 = fabs(thetaf + c), l4 = fabs(thetaf - c);
  if (!acoustics_clear(thetaf, c, thetaL, PL, L.ir, thetaR, PR, R.ir, gamma)) {
    const S cL = sqrt_s(gamma * PL * L.ir), cR = sqrt_s(gamma * PR * R.ir);
    l3 = entropy_fix(thetaf + c, thetaL + cL, thetaR + cR);
    l4 = entropy_fix(thetaf - c, thetaL - cL, thetaR - cR);
  }

  const S d0 = QR[0] - QL[0], d1 = QR[1] - QL[1], d2 = QR[2] - QL[2], d3 = QR[3] - QL[3], d4 = QR[4] - QL[4];

  // |A| dQ = T |L| Tinv dQ.  The three entropy/shear columns of T share the
  // eigenvalue l0, so the product is l0 dQ + (l3 - l0) P+ dQ + (l4 - l0) P- dQ
  // with P+/- the projectors on the two acoustic eigenvectors
  // r+/- = (1, u +/- c n, h +/- c theta): the same value as the reference's
  // two 5x5 products (any basis of the l0 eigenspace gives it), in about a
  // third of the operations.  P+/- dQ = a+/- r+/- with
  // a+/- = (dp +/- c rho dVn) / (2 c^2), where rho dVn = n.d(rho u) - theta d(rho)
  // and dp = (gamma - 1)(d(rho E) - u.d(rho u) + |u|^2/2 d(rho)) at the Roe state.
  const S rdvn = (nx * d1 + ny * d2 + nz * d3) - thetaf * d0;
  const S dp = gm1 * (d4 - (u * d1 + v * d2 + w * d3) + v2h * d0);
  const S hic2 = halve(ic2);
  const S ap3 = (l3 - l0) * ((dp + c * rdvn) * hic2);
  const S ap4 = (l4 - l0) * ((dp - c * rdvn) * hic2);
  const S sp = ap3 + ap4, sm = c * (ap3 - ap4);
  const S dr0 = l0 * d0 + sp;
  const S dr1 = l0 * d1 + (u * sp + nx * sm);
  const S dr2 = l0 * d2 + (v * sp + ny * sm);
  const S dr3 = l0 * d3 + (w * sp + nz * sm);
  const S dr4 = l0 * d4 + (h * sp + thetaf * sm);

  // physical fluxes (Flux, :686)
  const S ha = halve(area);
  flux[0] = ha * (L.rt + R.rt - dr0);
  flux[1] = ha * (L.f1 + R.f1 - dr1);
  flux[2] = ha * (L.f2 + R.f2 - dr2);
  flux[3] = ha * (L.f3 + R.f3 - dr3);
  flux[4] = ha * (hL * L.rt + hR * R.rt - dr4);
  const S zero = Sc<S>::c(0.0), tiny = Sc<S>::c(1.0e-10);
  return ((rL < zero || EL < tiny || PL < tiny) ? 1 : 0) | ((rR < zero || ER < tiny || PR < tiny) ? 2 : 0) |
         ((P < tiny || rE < tiny) ? 4 : 0);
}

// ---- FP64 forms ------------------------------------------------------------
// The FP64 pipe bounds every kernel that evaluates the flux in FP64 (88 % busy
// in the edge pass), so these specialisations take few FP64 instructions,
// about 160 an edge where the operators compile to 256: reciprocals, quotients
// and roots from FP32 seeds (seeded.cuh); the sides' acoustic speeds only
// where an FP32 test cannot rule the acoustic entropy fix out; halvings,
// selections and the non-physical tests on the integer pipes.  Every sum and
// product is rounded as in the operator form above with its multiply-adds
// fused left to right, so the flux is that form's bit for bit (but for one in
// 40,000 reciprocals, off by its last bit): the finite-difference Jacobian
// divides flux differences by 1e-8, and the FP32 Krylov solver rounds the
// residual, so both amplify a last bit by 1e8.
// Edge pass of the 128x96x96 box: 3.765 ms before, 2.366 ms now.

// x / 2, exact for any double: the exponent on the integer pipe
__device__ __forceinline__ double half_bits(double x) {
  if (!seed_range(abs_bits(x))) return 0.5 * x;
  return __hiloint2double(__double2hiint(x) - (1 << 20), __double2loint(x));
}

template <>
__device__ __forceinline__ RoeSide<double> roe_side_ir<double>(const double* Q, const double ir, const double nx,
                                                               const double ny, const double nz, const double gm1) {
  RoeSide<double> o;
  o.r = Q[0];
  o.ir = ir;
  o.u = __dmul_rn(Q[1], ir);
  o.v = __dmul_rn(Q[2], ir);
  o.w = __dmul_rn(Q[3], ir);
  o.E = Q[4];
  const double k2 = fma(o.w, o.w, fma(o.u, o.u, __dmul_rn(o.v, o.v)));
  o.P = __dmul_rn(gm1, fma(-half_bits(o.r), k2, o.E));
  o.h = __dmul_rn(__dadd_rn(o.E, o.P), ir);
  o.th = fma(o.w, nz, fma(o.u, nx, __dmul_rn(o.v, ny)));
  o.rt = __dmul_rn(o.r, o.th);
  o.f1 = fma(o.u, o.rt, __dmul_rn(o.P, nx));
  o.f2 = fma(o.v, o.rt, __dmul_rn(o.P, ny));
  o.f3 = fma(o.w, o.rt, __dmul_rn(o.P, nz));
  return o;
}

// |eig| with the Harten-Hyman fix (entropy_fix) for finite eigenvalues,
// selections on integer keys
__device__ __forceinline__ double entropy_fix64(double eig, double eigL, double eigR) {
  const double dl = __dsub_rn(eig, eigL), dr = __dsub_rn(eigR, eig);
  double eps = key_gt(dl, dr) ? dl : dr;
  if (!key_gt(eps, 0.0)) eps = 0.0;
  const double a = abs_bits(eig);
  return key_gt(eps, a) ? half_bits(__dadd_rn(quot(__dmul_rn(eig, eig), eps), eps)) : a;
}

template <FuseEnergy FUSE>
__device__ __forceinline__ int roe_core64(const RoeSide<double>& L, const RoeSide<double>& R,
                                          const RoePair<double>& pr, const double* QL, const double* QR,
                                          const double nx, const double ny, const double nz, const double area,
                                          const double gamma, const double gm1, const double igamma, double* flux) {
  // Roe-averaged state
  const double rho = pr.rho, sigma = pr.sigma;
  const double u = fma(sigma, __dsub_rn(R.u, L.u), L.u);
  const double v = fma(sigma, __dsub_rn(R.v, L.v), L.v);
  const double w = fma(sigma, __dsub_rn(R.w, L.w), L.w);
  const double h = fma(sigma, __dsub_rn(R.h, L.h), L.h);
  const double v2h = half_bits(fma(w, w, fma(u, u, __dmul_rn(v, v))));
  const double c2 = __dmul_rn(gm1, __dsub_rn(h, v2h));
  const double c = root(c2);
  const double ic2 = recip(c2);
  const double thetaf = fma(w, nz, fma(u, nx, __dmul_rn(v, ny)));

  // entropy-fixed |eigenvalues|
  const double l0 = entropy_fix64(thetaf, L.th, R.th);
  const double ep = __dadd_rn(thetaf, c), em = __dsub_rn(thetaf, c);
  double l3 = abs_bits(ep), l4 = abs_bits(em);
  if (!acoustics_clear(thetaf, c, L.th, L.P, L.ir, R.th, R.P, R.ir, gamma)) {
    const double cL = root(__dmul_rn(__dmul_rn(gamma, L.P), L.ir)), cR = root(__dmul_rn(__dmul_rn(gamma, R.P), R.ir));
    l3 = entropy_fix<double>(ep, __dadd_rn(L.th, cL), __dadd_rn(R.th, cR));
    l4 = entropy_fix<double>(em, __dsub_rn(L.th, cL), __dsub_rn(R.th, cR));
  }

  // |A| dQ in projector form
  const double d0 = __dsub_rn(QR[0], QL[0]), d1 = __dsub_rn(QR[1], QL[1]), d2 = __dsub_rn(QR[2], QL[2]),
               d3 = __dsub_rn(QR[3], QL[3]), d4 = __dsub_rn(QR[4], QL[4]);
  const double rdvn = fma(-thetaf, d0, fma(nz, d3, fma(nx, d1, __dmul_rn(ny, d2))));
  const double dp =
      __dmul_rn(gm1, fma(v2h, d0, __dsub_rn(d4, fma(w, d3, fma(u, d1, __dmul_rn(v, d2))))));
  const double hic2 = half_bits(ic2);
  const double k3 = __dsub_rn(l3, l0), k4 = __dsub_rn(l4, l0);
  const double t3 = __dmul_rn(fma(c, rdvn, dp), hic2);
  const double ap4 = __dmul_rn(k4, __dmul_rn(fma(-c, rdvn, dp), hic2));
  const double sp = fma(k3, t3, ap4), sm = __dmul_rn(c, fma(k3, t3, -ap4));
  const double dr0 = fma(l0, d0, sp);
  const double dr1 = fma(l0, d1, fma(u, sp, __dmul_rn(nx, sm)));
  const double dr2 = fma(l0, d2, fma(v, sp, __dmul_rn(ny, sm)));
  const double dr3 = fma(l0, d3, fma(w, sp, __dmul_rn(nz, sm)));
  const double dr4 = fma(l0, d4, fma(h, sp, __dmul_rn(thetaf, sm)));

  // physical fluxes (Flux, :686)
  const double ha = half_bits(area);
  flux[0] = __dmul_rn(ha, __dsub_rn(__dadd_rn(L.rt, R.rt), dr0));
  flux[1] = __dmul_rn(ha, __dsub_rn(__dadd_rn(L.f1, R.f1), dr1));
  flux[2] = __dmul_rn(ha, __dsub_rn(__dadd_rn(L.f2, R.f2), dr2));
  flux[3] = __dmul_rn(ha, __dsub_rn(__dadd_rn(L.f3, R.f3), dr3));
  const double fe = FUSE == FuseEnergy::left    ? fma(L.h, L.rt, __dmul_rn(R.h, R.rt))
                    : FUSE == FuseEnergy::right ? fma(R.h, R.rt, __dmul_rn(L.h, L.rt))
                                                : __dadd_rn(__dmul_rn(L.h, L.rt), __dmul_rn(R.h, R.rt));
  flux[4] = __dmul_rn(ha, __dsub_rn(fe, dr4));

  // BadExtrapolation of the three states.  The pressure and energy of the
  // Roe state are rho c2 / gamma and at least 1 / (gamma - 1) of it; all
  // clearly above the threshold, on the high words and for the product in
  // FP32, means no flag.
  const int lim = 0x3ddb7cdf;  // high word of 1e-10
  const bool clear = __double2hiint(L.r) >= 0 && __double2hiint(R.r) >= 0 && __double2hiint(L.E) > lim &&
                     __double2hiint(R.E) > lim && __double2hiint(L.P) > lim && __double2hiint(R.P) > lim &&
                     est_f32(rho) * est_f32(c2) > 1.0e-9f * est_f32(gamma) * (1.0f + est_f32(gm1));
  if (clear) return 0;
  const double zero = 0.0, tiny = 1.0e-10;
  const double rE = rho * igamma * (h + gm1 * v2h);
  const double P = gm1 * (rE - rho * v2h);
  return ((L.r < zero || L.E < tiny || L.P < tiny) ? 1 : 0) | ((R.r < zero || R.E < tiny || R.P < tiny) ? 2 : 0) |
         ((P < tiny || rE < tiny) ? 4 : 0);
}

// ComputeAuxiliaryVariables (ucs/compressible.tcc:1230) on a 10-wide FP64 record
__device__ __forceinline__ void aux_vars(double gamma, double* Q) {
  const double gm1 = gamma - 1.0;
  const double ir = recip(Q[0]);
  const double u = Q[1] * ir, v = Q[2] * ir, w = Q[3] * ir;
  const double P = gm1 * (Q[4] - 0.5 * Q[0] * (u * u + v * v + w * w));
  Q[6] = P;
  Q[5] = gamma * P * ir;
  Q[7] = u;
  Q[8] = v;
  Q[9] = w;
}

// Sutherland's law (EqnSet::ComputeViscosity, ucs/eqnset.h:251)
template <class S>
__device__ __forceinline__ S sutherland(S T, S S_) {
  return div_s((Sc<S>::c(1.0) + S_) * (T * sqrt_s(T)), T + S_);
}

// ViscousFlux (ucs/compressible.tcc:713) for laminar flow (mut = 0).
// (u, v, w, T): the face-averaged state; grad: 27-wide face gradient;
// rk = area / ReTilde.
template <class S>
__device__ __forceinline__ void viscous_flux(const S u, const S v, const S w, const S T, const S* grad, const S nx,
                                             const S ny, const S nz, const S rk, const S Sconst, const S cp_over_pr,
                                             S* flux) {
  const S Tx = grad[15], Ty = grad[16], Tz = grad[17];
  const S ux = grad[18], uy = grad[19], uz = grad[20];
  const S vx = grad[21], vy = grad[22], vz = grad[23];
  const S wx = grad[24], wy = grad[25], wz = grad[26];
  const S two = Sc<S>::c(2.0);
  const S mu = sutherland(T, Sconst);
  const S fact = Sc<S>::c(-2.0 / 3.0) * (ux + vy + wz);
  const S tauxx = twice(ux) + fact, tauyy = twice(vy) + fact, tauzz = twice(wz) + fact;
  const S tauxy = uy + vx, tauxz = uz + wx, tauyz = vz + wy;
  const S RKT = rk * mu;
  const S c1 = -(mu * cp_over_pr);
  const S Tn = Tx * nx + Ty * ny + Tz * nz;
  const S tauxn = tauxx * nx + tauxy * ny + tauxz * nz;
  const S tauyn = tauxy * nx + tauyy * ny + tauyz * nz;
  const S tauzn = tauxz * nx + tauyz * ny + tauzz * nz;
  flux[0] = Sc<S>::c(0.0);
  flux[1] = -RKT * tauxn;
  flux[2] = -RKT * tauyn;
  flux[3] = -RKT * tauzn;
  flux[4] = -RKT * (tauxn * u + tauyn * v + tauzn * w) + rk * c1 * Tn;
}

}  // namespace pcfd
