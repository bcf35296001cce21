// thx_face.cuh -- FP64 surface fluxes with shared reciprocals (ideal gas).
//
// The surface fluxes of thx_device.cuh divide twelve to twenty times per face
// point, nearly always by the density of one side: at 40^3 p=3 the LLF face
// kernel spent 70 % of its issue slots and four fifths of its time on them.
// With density and pressure of both sides in the range of the shared
// reciprocals (thx_volume.cuh) one reciprocal per side serves them all; the
// operations and their order are those of thx_device.cuh, and so the results.
#pragma once

namespace thx {

template <int DIM>
struct FaceSide {
  double q[DIM + 2], v[DIM], p, yr;  // conserved state, velocity, pressure, ~1/rho
  bool ok;                           // density and pressure in range
};

template <int DIM>
__device__ __forceinline__ void face_side(const GasT<double> &g, const double *q, FaceSide<DIM> &s) {
  double m2 = 0.0;
#pragma unroll
  for (int k = 0; k < DIM + 2; ++k) s.q[k] = q[k];
  s.yr = rcp_refined(q[0]);
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    m2 += q[1 + d] * q[1 + d];
    s.v[d] = div_by(q[1 + d], q[0], s.yr);
  }
  s.p = g.gm1 * (q[DIM + 1] - div_by(0.5 * m2, q[0], s.yr));
  s.ok = in_fast_range(q[0]) && in_fast_range(s.p);
}

// a / b for several a: by the reciprocal of b where b is in range
struct SharedDiv {
  double b, y;
  bool ok;
  __device__ __forceinline__ explicit SharedDiv(double x) : b(x), y(rcp_refined(x)), ok(in_fast_range(x)) {}
  __device__ __forceinline__ double operator()(double a) const { return ok ? div_by(a, b, y) : a / b; }
};

// Fluxes that have a shared form.
__host__ __device__ constexpr bool surf_shared(int surf) {
  return surf == SURF_CHANDRASHEKAR || surf == SURF_HLL || surf == SURF_LLF || surf == SURF_ROE;
}

// surface_flux<double, DIM, SURF> of thx_device.cuh.
template <int DIM, int SURF>
__device__ __forceinline__ void surface_flux_shared(const GasT<double> &g, const FaceSide<DIM> &A,
                                                    const FaceSide<DIM> &B, const double *n, double *F) {
  constexpr int E = DIM + 1;
  const double *q1 = A.q, *q2 = B.q;
  if constexpr (SURF == SURF_CHANDRASHEKAR) {
    const double beta1 = div_by(0.5 * q1[0], A.p, rcp_refined(A.p)), beta2 = div_by(0.5 * q2[0], B.p, rcp_refined(B.p));
    const LogMeans m = log_means<LM_BRANCH>(q1[0], q2[0], beta1, beta2);
    const double rho_mean = 0.5 * (q1[0] + q2[0]), drho = q2[0] - q1[0];
    double mom[DIM], hhat = 0.0, vn = 0.0, vn1 = 0.0, vn2 = 0.0, nor = 0.0, de = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const double v1 = A.v[d], v2 = B.v[d], vbar = 0.5 * (v1 + v2);
      vn += vbar * n[d];
      mom[d] = m.a * vbar;
      hhat += -0.25 * (v1 * v1 + v2 * v2) + vbar * vbar;
      nor += n[d] * n[d];
      vn1 += v1 * n[d];
      vn2 += v2 * n[d];
      de += 0.5 * drho * v1 * v2 + rho_mean * (v2 - v1) * vbar;
    }
    const double p_hat = div_by(0.5 * (q1[0] + q2[0]), m.s2, m.rs2);
    hhat += div_by(0.5, m.b, m.ib) * g.gm1_av_inv + div_by(p_hat, m.a, m.ia);
    // scalar dissipation
    nor = sqrt(nor);
    const double lmax = rmax(rabs(vn1) + sqrt(div_by(g.gamma * A.p, q1[0], A.yr)) * nor,
                             rabs(vn2) + sqrt(div_by(g.gamma * B.p, q2[0], B.yr)) * nor);
    const double ib1 = div_by(1.0, beta1, rcp_refined(beta1)), ib2 = div_by(1.0, beta2, rcp_refined(beta2));
    de += div_by(0.5 * drho * g.inv_gm1, m.b, m.ib) + 0.5 * rho_mean * g.inv_gm1 * (ib2 - ib1);
    F[0] = m.a * vn - 0.5 * lmax * drho;
#pragma unroll
    for (int d = 0; d < DIM; ++d) F[1 + d] = vn * mom[d] + p_hat * n[d] - 0.5 * lmax * (q2[1 + d] - q1[1 + d]);
    F[E] = m.a * vn * hhat - de * (0.5 * lmax);
    return;
  }
  NState<double, DIM> L, R;
  L.inv_rho = div_by(1.0, q1[0], A.yr);
  R.inv_rho = div_by(1.0, q2[0], B.yr);
  L.p = L.pp = A.p;
  R.p = R.pp = B.p;
  L.H = (q1[E] + A.p) * L.inv_rho;
  R.H = (q2[E] + B.p) * R.inv_rho;
  double un1 = 0.0, un2 = 0.0, nn = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    un1 += A.v[d] * n[d];
    un2 += B.v[d] * n[d];
    nn += n[d] * n[d];
  }
  const double nm = sqrt(nn);
  if constexpr (SURF == SURF_HLL) {
    const double c1 = sqrt(div_by(g.gamma * A.p, q1[0], A.yr)) * nm, c2 = sqrt(div_by(g.gamma * B.p, q2[0], B.yr)) * nm;
    const double sL1 = un1 - c1, sL2 = un2 - c2, sR1 = un1 + c1, sR2 = un2 + c2;
    const double sL = (sL1 < sL2) ? sL1 : sL2;
    const double sR = (sR1 > sR2) ? sR1 : sR2;
    const SharedDiv over(sR - sL);
#pragma unroll
    for (int e = 0; e < DIM + 2; ++e) {
      const double fn1 = normal_flux<double, DIM>(q1, L, n, e), fn2 = normal_flux<double, DIM>(q2, R, n, e);
      if (sL >= 0.0) F[e] = fn1;
      else if (sR <= 0.0) F[e] = fn2;
      else F[e] = over(sR * fn1 - sL * fn2 + sL * sR * (q2[e] - q1[e]));
    }
  } else if constexpr (SURF == SURF_LLF) {
    const double lmax = rmax(rabs(un1) + sqrt(div_by(g.gamma * A.p, q1[0], A.yr)) * nm,
                             rabs(un2) + sqrt(div_by(g.gamma * B.p, q2[0], B.yr)) * nm);
#pragma unroll
    for (int e = 0; e < DIM + 2; ++e) {
      const double nl = normal_flux<double, DIM>(q1, L, n, e), nr = normal_flux<double, DIM>(q2, R, n, e);
      F[e] = 0.5 * (nl + nr) - 0.5 * lmax * (q2[e] - q1[e]);
    }
  } else {
    const double inv_nm = 1.0 / nm;
    const double rootL = sqrt(q1[0]), rootR = sqrt(q2[0]);
    const double sum = rootL + rootR;
    const double rsi = div_by(1.0, sum, rcp_refined(sum));
    const double rho_roe = rootL * rootR;
    const double HL = div_by(q1[E] + A.p, q1[0], A.yr), HR = div_by(q2[E] + B.p, q2[0], B.yr);
    const double H = (rootL * HL + rootR * HR) * rsi;
    double u[DIM], du_t[DIM], nh[DIM], du[DIM];
    double u2 = 0.0, un = 0.0, dun = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const double uL = A.v[d], uR = B.v[d];
      nh[d] = n[d] * inv_nm;
      u[d] = (rootL * uL + rootR * uR) * rsi;
      du[d] = uR - uL;
      u2 += u[d] * u[d];
      un += u[d] * nh[d];
      dun += du[d] * nh[d];
    }
    const double a2 = (g.gamma - 1.0) * (H - 0.5 * u2);
    const double a = sqrt(a2);
    const SharedDiv over(a2);
    const double dp = B.p - A.p, drho = q2[0] - q1[0];
    const double am = over(0.5 * (dp - rho_roe * a * dun));
    const double ap = over(0.5 * (dp + rho_roe * a * dun));
    const double az = drho - over(dp);
    const double lm = rabs(un - a) * nm, lz = rabs(un) * nm, lp = rabs(un + a) * nm;
#pragma unroll
    for (int d = 0; d < DIM; ++d) du_t[d] = du[d] - dun * nh[d];
    double diss[DIM + 2];
    diss[0] = lm * am + lz * az + lp * ap;
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      diss[1 + d] = lm * am * (u[d] - a * nh[d]) + lz * (az * u[d] + rho_roe * du_t[d]) + lp * ap * (u[d] + a * nh[d]);
    double udt = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) udt += u[d] * du_t[d];
    diss[E] = lm * am * (H - a * un) + lz * (0.5 * az * u2 + rho_roe * udt) + lp * ap * (H + a * un);
#pragma unroll
    for (int e = 0; e < DIM + 2; ++e)
      F[e] = 0.5 * (normal_flux<double, DIM>(q1, L, n, e) + normal_flux<double, DIM>(q2, R, n, e)) - 0.5 * diss[e];
  }
}

// F* of the states qm, qp (stored form) along n, where the surface flux has a
// shared form and both states are in its range.
template <int DIM, int SURF>
__device__ __forceinline__ bool try_surface_flux_shared(const GasT<double> &g, const int kind, const double *qm,
                                                        const double *qp, const double *n, double *F) {
  if (SURF >= 0 ? !surf_shared(SURF) : !surf_shared(kind)) return false;
  FaceSide<DIM> A, B;
  face_side<DIM>(g, qm, A);
  face_side<DIM>(g, qp, B);
  if (!A.ok || !B.ok) return false;
  if constexpr (SURF >= 0) {
    if constexpr (surf_shared(SURF)) surface_flux_shared<DIM, SURF>(g, A, B, n, F);
  } else {
    switch (kind) {
      case SURF_CHANDRASHEKAR: surface_flux_shared<DIM, SURF_CHANDRASHEKAR>(g, A, B, n, F); break;
      case SURF_HLL: surface_flux_shared<DIM, SURF_HLL>(g, A, B, n, F); break;
      case SURF_LLF: surface_flux_shared<DIM, SURF_LLF>(g, A, B, n, F); break;
      default: surface_flux_shared<DIM, SURF_ROE>(g, A, B, n, F); break;
    }
  }
  return true;
}

}  // namespace thx
