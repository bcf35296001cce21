// thx_volume.cuh -- flux-differencing volume kernel of the ideal gas: one
// thread per tensor line.
//
// What bounds it: the arithmetic pipes (FP64: 60 % of the pipe's cycles at
// 20^3 p=4, with 43 % of the issue slots; FP32: 64 % of the issue slots).  A
// thread owns a line of N nodes: it evaluates the line's N(N-1)/2 symmetric
// pairs once each and adds every pair flux to its two end nodes.  Against one
// thread per pair, with the fluxes passed through shared memory to one thread
// per node (15 shared-memory accesses and their index arithmetic per pair),
// it executes a third of the instructions: at 32^3 p=4 Ranocha, with the
// shared reciprocals below, 0.712 -> 0.357 ms in FP64 and 0.370 -> 0.171 ms
// FP32-mixed (less the viscous divergence, which the gradient kernel forms).
// Pairs run in (lower, upper) lexicographic order, so every node receives its
// terms in the order of the other end's index, as
// include/DGSEMIntegrator.hpp:147-164 sums them, and the sums of the
// directions continue one another through shared memory.  The thread of a
// line of the last direction holds finished columns and goes on to the
// surface lift and the Runge-Kutta stage.
#pragma once
#include <type_traits>

namespace thx {

template <int DIM, int N, int T, int EPBX = 0>
struct LineShape {
  static constexpr int ND = DIM == 2 ? N * N : N * N * N;
  static constexpr int NFP = ND / N;
  static constexpr int NL = ND / N;        // lines per direction
  static constexpr int NEQ = DIM + 2;
  static constexpr int THREADS = T;
  // elements per CTA: as many as have a thread for every line, or EPBX
  static constexpr int EPB = EPBX > 0 ? EPBX : T / NL;
  static_assert(EPB >= 1 && EPB * NL <= T, "a thread for every line");
  // x-lines are an odd number of words apart, so that the threads of
  // neighbouring x-lines read different banks
  static constexpr int LS = N % 2 ? N : N + 1;
  static constexpr int NDP = LS * NL;      // padded nodes per element
  static constexpr int FS = EPB * NDP;     // stride of a field
};

// Threads per CTA of the line kernels: 128 (3-D: 3 to 14 elements; three or
// more CTAs per SM, see line_min_blocks).
constexpr int kLineThreads = 128;

// NODAL: the metric varies within the element and is read from memory;
// otherwise one metric per element, staged.
template <typename R, int DIM, int N, int VOL, int T, int EPBX = 0, bool NODAL = false>
struct LineSmem {
  using S = LineShape<DIM, N, T, EPBX>;
  static constexpr int PRIM = node_fields<R, DIM, VOL>();
  static constexpr int FIELDS = PRIM + S::NEQ;
  static constexpr int OPS = (N * N + 1) / 2 * 2;
  static constexpr int MET = NODAL ? 0 : (S::EPB * DIM * DIM + 1) / 2 * 2;
  static constexpr size_t bytes() {
    return sizeof(R) * ((size_t)OPS + MET + (size_t)FIELDS * S::FS) + sizeof(int) * S::EPB * 2 * DIM;
  }
};

// ---- FP64 pair fluxes with shared reciprocals ------------------------------
// An FP64 division costs a reciprocal refinement, a residual correction and a
// range test; the Ranocha and Chandrashekar fluxes have seven and nine per
// pair.  Their denominators are few: with every density and pressure of the
// CTA between 2^-100 and 2^100 (tested once per node), one reciprocal of
// their product serves both logarithmic means, and each quotient is rounded
// from it by the residual correction q + (a - b q) y (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990).  From y = (1 + d)/b the corrected quotient is off by at
// most |d| (2^53 |d| + 1) ulp before its rounding, below 2^-34 ulp for the
// least accurate reciprocal used (4e-14): it is the correctly rounded a / b
// but for quotients that close to a rounding boundary.  Everything else -- the
// branch variable, the series, the logarithm -- is formed as log_mean and the
// fluxes of thx_device.cuh form it, so the results do not depend on which of
// the two a CTA takes.  (The branch variable from a reciprocal instead of a
// quotient, and the series with fused multiply-adds, would be up to 3 % faster
// and change the last bit of about one mean in 10^4.)

// log_mean(x, y) and its reciprocal (to a few ulp, for div_by), given
// rx ~ 1/x, s = x + y and rs ~ 1/s.
template <int MODE>
__device__ __forceinline__ void log_mean_rcp(double x, double y, double s, double rx, double rs, double &lm,
                                             double &inv) {
  const double xi = div_by(y, x, rx);
  const double v = x * rs;  // 1/(xi + 1)
  const double u = div_by(xi * (xi - 2.0) + 1.0, xi * (xi + 2.0) + 1.0, v * v);
  if (MODE == LM_SERIES || u < 1e-4) {
    const double z = u * (35.0 + u * (21.0 + 15.0 * u));
    const double denom = 105.0 + z;
    // 1/denom from its expansion about 1/105 (z < 0.0036: to 4e-14)
    constexpr double c = 1.0 / 105.0;
    lm = div_by(s * 52.5, denom, __fma_rn(z, __fma_rn(z, c * c * c, -c * c), c));
    inv = denom * (rs * (1.0 / 52.5));
  } else {
    const double d = y - x, l = log_normal(xi);
    const double r = rcp_refined(l * d);
    lm = div_by(d, l, r * d);
    inv = l * (r * l);
  }
}

// Both logarithmic means of a pair, (x1, y1) and (x2, y2), and 1/(x2 + y2).
struct LogMeans {
  double a, ia, b, ib, s2, rs2;
};
template <int MODE>
__device__ __forceinline__ LogMeans log_means(double x1, double y1, double x2, double y2) {
  LogMeans m;
  const double s1 = x1 + y1, s2 = x2 + y2;
  const double p1 = x1 * s1, p2 = x2 * s2;
  const double r = rcp_refined(p1 * p2);
  const double r1 = r * p2, r2 = r * p1;
  m.s2 = s2;
  m.rs2 = r2 * x2;
  log_mean_rcp<MODE>(x1, y1, s1, r1 * s1, r1 * x1, m.a, m.ia);
  log_mean_rcp<MODE>(x2, y2, s2, r2 * s2, m.rs2, m.b, m.ib);
  return m;
}

// vol_chandrashekar and vol_ranocha with the shared reciprocals: the same
// operations in the same order.
template <int DIM, int MODE>
__device__ __forceinline__ void pair_chandrashekar(const GasT<double> &g, const double *a, const double *b,
                                                   const double *met, double *F) {
  const LogMeans m = log_means<MODE>(a[0], b[0], a[DIM + 2], b[DIM + 2]);
  double mom[DIM], h = 0.0, vn = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const double v1 = a[1 + d], v2 = b[1 + d];
    const double vbar = 0.5 * (v1 + v2);
    vn += vbar * met[d];
    mom[d] = m.a * vbar;
    h += -0.25 * (v1 * v1 + v2 * v2) + vbar * vbar;
  }
  const double p_hat = div_by(0.5 * (a[0] + b[0]), m.s2, m.rs2);
  h += div_by(0.5, m.b, m.ib) * g.gm1_av_inv + div_by(p_hat, m.a, m.ia);
  F[0] = m.a * vn;
#pragma unroll
  for (int d = 0; d < DIM; ++d) F[1 + d] = vn * mom[d] + p_hat * met[d];
  F[DIM + 1] = m.a * vn * h;
}

template <int DIM, int MODE>
__device__ __forceinline__ void pair_ranocha(const GasT<double> &g, const double *a, const double *b,
                                             const double *met, double *F) {
  const double p1 = a[DIM + 1], p2 = b[DIM + 1];
  const LogMeans m = log_means<MODE>(a[0], b[0], a[0] * p2, b[0] * p1);
  const double pbar = 0.5 * (p1 + p2);
  double vbar[DIM], ke = 0.0, vn = 0.0, fe = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const double v1 = a[1 + d], v2 = b[1 + d];
    vbar[d] = 0.5 * (v1 + v2);
    vn += vbar[d] * met[d];
    ke += 0.5 * (v1 * v2);
    fe += (0.5 * (p1 * v2 + p2 * v1)) * met[d];
  }
  const double ie = div_by(p1 * p2, m.b, m.ib) * g.inv_gm1;
  F[0] = m.a * vn;
#pragma unroll
  for (int d = 0; d < DIM; ++d) F[1 + d] = m.a * vn * vbar[d] + pbar * met[d];
  F[DIM + 1] = fe + m.a * (ie + ke) * vn;
}

// The two-point flux of a pair.  SHARED: with the shared reciprocals (FP64;
// every density and pressure in their range).
template <typename R, int DIM, int VOL, bool SHARED, int MODE>
__device__ __forceinline__ void pair_flux(const GasT<R> &g, const R *A, const R *B, const R *met, R *F) {
  if constexpr (SHARED && VOL == VOL_CHANDRASHEKAR) pair_chandrashekar<DIM, MODE>(g, A, B, met, F);
  else if constexpr (SHARED && VOL == VOL_RANOCHA) pair_ranocha<DIM, MODE>(g, A, B, met, F);
  else if constexpr (VOL == VOL_CHANDRASHEKAR) vol_chandrashekar<R, DIM, MODE>(g, A, B, met, F);
  else if constexpr (VOL == VOL_RANOCHA) vol_ranocha<R, DIM, MODE>(g, A, B, met, F);
  else if constexpr (VOL == VOL_PIROZZOLI) vol_pirozzoli<R, DIM>(g, A, B, met, F);
  else vol_central<R, DIM>(A, B, met, F);
}

// Whether every logarithmic mean between the nodes of a line takes its
// series: the largest ratio of its arguments over the line stays below the
// branch's (ratio 1.0202 for ((r-1)/(r+1))^2 < 1e-4 in FP64, 1.105 for 2.5e-3
// in FP32, 1.666 for 1/16 in the perturbation form).
template <typename R, int DIM, int N, int VOL, int FS>
__device__ __forceinline__ bool series_line(const GasT<R> &g, const R *sP, int base, int stride) {
  if (VOL != VOL_CHANDRASHEKAR && VOL != VOL_RANOCHA) return true;
  // Chandrashekar's means are of the density and of beta, Ranocha's of the
  // density and of the cross products of density and pressure
  bool pert = false;
  if constexpr (IsF32<R>::value) pert = VOL == VOL_CHANDRASHEKAR && g.pert;
  const int second = VOL == VOL_CHANDRASHEKAR && !pert ? DIM + 2 : DIM + 1;
  R lo[2], hi[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const R *f = sP + (q == 0 ? 0 : second * FS) + base;
    lo[q] = hi[q] = f[0];
#pragma unroll
    for (int i = 1; i < N; ++i) {
      const R x = f[i * stride];
      lo[q] = x < lo[q] ? x : lo[q];
      hi[q] = x > hi[q] ? x : hi[q];
    }
  }
  const R bound = pert ? R(1.65) : IsF32<R>::value ? R(1.10) : R(1.0195);
  if (VOL == VOL_RANOCHA) return lo[0] > R(0) && lo[1] > R(0) && hi[0] * hi[1] < bound * (lo[0] * lo[1]);
  return lo[0] > R(0) && lo[1] > R(0) && hi[0] < bound * lo[0] && hi[1] < bound * lo[1];
}

// 2^-100 <= x < 2^100 (false for x <= 0 and NaN)
__device__ __forceinline__ bool in_fast_range(double x) {
  return (unsigned)(__double2hiint(x) - 0x39B00000) < 0x0C800000u;
}

// First padded node and node stride of a line.
template <int DIM, int N, int LS>
__device__ __forceinline__ void line_base(int dir, int line, int &base, int &stride) {
  if (dir == 0) {
    base = LS * line;
    stride = 1;
  } else if (DIM == 2) {
    base = line;
    stride = LS;
  } else if (dir == 1) {
    base = (line % N) + LS * N * (line / N);
    stride = LS;
  } else {
    base = (line % N) + LS * (line / N);
    stride = LS * N;
  }
}

// entropy_vars (thx_device.cuh) with the seven quotients formed from two
// reciprocals where density and pressure are in their range: the same
// operations in the same order.
template <int DIM>
__device__ __forceinline__ void entropy_vars_shared(const GasT<double> &g, const double *q, double *w) {
  const double rho = q[0];
  double m2 = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) m2 += q[1 + d] * q[1 + d];
  const double yr = rcp_refined(rho);
  const double ke = div_by(0.5 * m2, rho, yr);
  const double p = g.gm1 * (q[DIM + 1] - ke);
  if (!in_fast_range(rho) || !in_fast_range(p)) {
    entropy_vars<double, DIM>(g, q, w);
    return;
  }
  const double s = rlog(p) - g.gamma * rlog(rho);
  const double beta = div_by(rho, p, rcp_refined(p));
  w[0] = div_by(g.gamma - s, g.gamma - 1.0, g.inv_gm1) - beta * div_by(ke, rho, yr);
#pragma unroll
  for (int d = 0; d < DIM; ++d) w[1 + d] = beta * div_by(q[1 + d], rho, yr);
  w[DIM + 1] = -beta;
}

// Lift weight of face point fp of an elem_face entry; zero (and false) without
// an interior face.
template <typename R, int DIM, int NFP>
__device__ __forceinline__ bool lift_weight(const VolArgs<R> &a, const int fs, const int fp, R &w) {
  const int face = fs >> 1, side = fs & 1;
  const bool in = fs >= 0 && (IsF32<R>::value || !a.bw || face < a.nf_int);
  w = R(0);
  if (in) w = (side == 0 ? a.wm : a.wp)[(long long)face * a.w_fs + (long long)fp * a.w_ps];
  if (side == 0) w = -w;
  return in;
}

// Node n of element e from its sum du of the volume terms: scale by -1/J (sc
// = 1/J), blend (al: the element's coefficient), viscous divergence, surface
// lift -- the node's faces f[DIM] (elem_face entries, one per direction, or
// negative) at points fp with interior weights w and fluxes fl -- and the
// rate or the Runge-Kutta stage.
template <typename R, int DIM, int N>
__device__ __forceinline__ void finish_node(const VolArgs<R> &a, const int e, const int n, const R sc,
                                            const double al, const double dt, const int *f, const int *fp,
                                            const R *w, const R (*fl)[DIM + 2], R *du, bool &bad) {
  constexpr int ND = DIM == 2 ? N * N : N * N * N, NEQ = DIM + 2;
  const long long L = (long long)a.ne * ND, gi = (long long)e * ND + n;
  R dv[NEQ - 1];
#pragma unroll
  for (int k = 0; k < NEQ - 1; ++k) {
    dv[k] = R(0);
    if (a.vdiv) dv[k] = a.vdiv[k * L + gi];
  }
#pragma unroll
  for (int k = 0; k < NEQ; ++k) du[k] = -sc * du[k];
  // subcell finite-volume blend (include/EulerOperator_impl.hpp:134-152):
  // fv_kernel has stored the FV rate of every blended element
  if (al > 1e-16) {
    const R af = (R)al, ad = (R)(1.0 - al);
#pragma unroll
    for (int k = 0; k < NEQ; ++k) du[k] = ad * du[k] + af * a.fvrate[((long long)e * NEQ + k) * ND + n];
  }
  // divergence of the viscous flux (its mass row is zero), from the gradient
  // kernel
  if (a.vdiv) {
#pragma unroll
    for (int k = 0; k < NEQ - 1; ++k) du[1 + k] += sc * dv[k];
  }
  lift_and_store<R, DIM, N>(a, e, n, dt, f, fp, w, fl, du, bad);
}

// The last of finish_node: the surface lift of du, and the rate or the
// Runge-Kutta stage.
template <typename R, int DIM, int N>
__device__ __forceinline__ void lift_and_store(const VolArgs<R> &a, const int e, const int n, const double dt,
                                               const int *f, const int *fp, const R *w, const R (*fl)[DIM + 2], R *du,
                                               bool &bad) {
  constexpr int ND = DIM == 2 ? N * N : N * N * N, NFP = ND / N, NEQ = DIM + 2;
  const long long L = (long long)a.ne * ND, gi = (long long)e * ND + n;
  // interior faces summed first, then added (restr_f transpose; +=); then the
  // boundary faces the same way (restr_b)
#pragma unroll
  for (int k = 0; k < NEQ; ++k) {
    R sum = R(0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) sum += w[d] * fl[d][k];
    du[k] += sum;
  }
  if constexpr (!IsF32<R>::value) {
    if (a.bw) {
      R sum[NEQ];
#pragma unroll
      for (int k = 0; k < NEQ; ++k) sum[k] = R(0);
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        const int face = f[d] >> 1;
        if (f[d] < 0 || face < a.nf_int) continue;
        const R wb = -a.bw[(long long)(face - a.nf_int) * NFP + fp[d]];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) sum[k] += wb * a.fstar[((long long)face * NEQ + k) * NFP + fp[d]];
      }
#pragma unroll
      for (int k = 0; k < NEQ; ++k) du[k] += sum[k];
    }
  }
  if (a.stage == 0) {
    if (a.du64) {
#pragma unroll
      for (int k = 0; k < NEQ; ++k) a.du64[k * L + gi] = (double)du[k];
    } else {
#pragma unroll
      for (int k = 0; k < NEQ; ++k) a.du[k * L + gi] = du[k];
    }
    return;
  }
  // fused SSP-RK3 stage in the arithmetic order of mfem::RK3SSPSolver::Step;
  // every load before the first store.  A device-side step of 0 (a finished
  // time loop, or no valid rate) leaves the state exactly as it was.
  const bool still = a.dt_dev && dt == 0.0;
  double umv[NEQ], yv[NEQ];
#pragma unroll
  for (int k = 0; k < NEQ; ++k) {
    umv[k] = a.um[k * L + gi];
    yv[k] = a.stage == 1 ? 0.0 : a.y[k * L + gi];
  }
  double ynew[NEQ];
#pragma unroll
  for (int k = 0; k < NEQ; ++k) {
    const double kk = (double)du[k];
    double y;
    if (a.stage == 1) {
      y = umv[k] + dt * kk;
    } else if (a.stage == 2) {
      y = yv[k] + dt * kk;
      y = 0.75 * umv[k] + 0.25 * y;
    } else {
      y = yv[k] + dt * kk;
      y = (1.0 / 3.0) * umv[k] + (2.0 / 3.0) * y;
      if (still) y = umv[k];
    }
    ynew[k] = y;
  }
#pragma unroll
  for (int k = 0; k < NEQ; ++k) {
    const long long g = k * L + gi;
    if (a.stage == 3) {
      if (!still) a.um[g] = ynew[k];
    } else {
      a.yo[g] = ynew[k];
    }
    if (a.yf) a.yf[g] = (float)(ynew[k] - a.off[k]);
  }
  if constexpr (IsF32<R>::value) {
    // FP32-mixed: positivity of the new FP64 stage state, in FP64
    if (!fp64_state_positive<DIM>(ynew, (double)a.gas.gm1)) bad = true;
  }
}

// One CTA's work: elements [block*EPB, block*EPB + EPB).  su: the block's
// state staged in shared memory (array k at k*kstride), or nullptr.  Without
// NODAL the metric must be one per element (met_ns == 0).
template <typename R, int DIM, int N, int VOL, int T, int EPBX = 0, bool NODAL = false>
__device__ __forceinline__ void volume_line_body(const VolArgs<R> &a, const int block, const R *su = nullptr,
                                                 const int kstride = 0) {
  using S = LineShape<DIM, N, T, EPBX>;
  using M = LineSmem<R, DIM, N, VOL, T, EPBX, NODAL>;
  constexpr int ND = S::ND, NEQ = S::NEQ, EPB = S::EPB, NL = S::NL, FS = S::FS, PRIM = M::PRIM;
  constexpr bool FASTABLE = !IsF32<R>::value && (VOL == VOL_CHANDRASHEKAR || VOL == VOL_RANOCHA);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (dynamic_smem_bytes() < M::bytes()) {
    if (threadIdx.x == 0) atomicOr(a.status, STATUS_LAUNCH);
    return;
  }
  R *sD = reinterpret_cast<R *>(smem_raw);  // Dhat2
  R *sM = sD + M::OPS;                      // [EPB][DIM][DIM] metric rows (one per element)
  R *sP = sM + M::MET;                      // [PRIM][EPB][NDP] node data
  R *sR = sP + PRIM * FS;                   // [NEQ][EPB][NDP] sums of the directions so far
  int *sF = reinterpret_cast<int *>(sR + NEQ * FS);  // [EPB][2*DIM] elem_face
  const int tid = threadIdx.x;
  const int e0 = block * EPB;
  const long long L = (long long)a.ne * ND;
  const int nodes = min(EPB, a.ne - e0) * ND;
  // node data: every load of the thread's nodes is issued before the first use
  constexpr int IT = (EPB * ND + T - 1) / T;
  R qn[IT][NEQ];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int i = tid + it * T;
#pragma unroll
    for (int k = 0; k < NEQ; ++k) {
      if (su) qn[it][k] = i < nodes ? su[k * kstride + i] : R(1);
      else qn[it][k] = i < nodes ? a.u[k * L + (long long)e0 * ND + i] : R(1);
    }
  }
  for (int i = tid; i < N * N; i += T) sD[i] = a.ops[i];
  for (int i = tid; i < nodes / ND * 2 * DIM; i += T) sF[i] = a.elem_face[(long long)e0 * 2 * DIM + i];
  if constexpr (!NODAL) {
    for (int i = tid; i < nodes / ND * DIM * DIM; i += T)
      sM[i] = a.met[(long long)(e0 + i / (DIM * DIM)) * a.met_es + i % (DIM * DIM)];
  }
  bool slow = false;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int i = tid + it * T;
    R pr[nprim<R, DIM>()], fl[PRIM];
    const R *q = qn[it];
    if (i >= nodes) continue;
    node_prims<R, DIM, VOL>(a.gas, q, pr);
    pack_node<R, DIM, VOL>(a.gas, q, pr, fl);
    const int pn = i + (N % 2 ? 0 : i / N);
#pragma unroll
    for (int k = 0; k < PRIM; ++k) sP[k * FS + pn] = fl[k];
    if constexpr (!IsF32<R>::value) {
      // FP64 path: positivity of the state read here.  FP32-mixed: checked
      // on the FP64 master state instead (to_working, the RK stage epilogue)
      if (!(pr[0] > R(0)) || !(pr[DIM + 1] > R(0))) atomicOr(a.status, STATUS_NONPOSITIVE);
      if constexpr (FASTABLE) slow = slow || !in_fast_range(pr[0]) || !in_fast_range(pr[DIM + 1]);
    }
  }
  if constexpr (FASTABLE) slow = __syncthreads_or(slow);
  else __syncthreads();

  const int el = tid / NL, line = tid - el * NL;
  const int e = e0 + el;
  bool active = el < EPB && e < a.ne;
  // FP32-mixed with FP64 islands: elements that the FP64 kernels evaluate
  if (active && a.skip_block) active = a.skip_block[e / a.skip_epb] == 0;
  // The column of the last direction: its faces in the other directions (one
  // of a pair, or none) and the two at its ends
  const int cx = line % N, cy = DIM == 3 ? line / N : 0;
  int fd[DIM + 1];
#pragma unroll
  for (int d = 0; d < DIM + 1; ++d) {
    const int c = d == 0 ? cx : cy;
    const int lf = d < DIM - 1 ? 2 * d + (c == N - 1 ? 1 : 0) : 2 * (DIM - 1) + (d - (DIM - 1));
    fd[d] = active && (d >= DIM - 1 || c == 0 || c == N - 1) ? sF[el * 2 * DIM + lf] : -1;
  }
  const double al = active && a.alpha ? a.alpha[e] : 0.0;
  const R *jac = a.jac + (long long)e * a.jac_es + (long long)line * a.jac_ns;
  R sc = active ? R(1) / jac[0] : R(1);
  const double dt = a.stage == 0 ? 0.0 : a.dt_dev ? *a.dt_dev : a.dt;
  bool bad = false;

#pragma unroll 1
  for (int dir = 0; dir < DIM; ++dir) {
    const bool last = dir == DIM - 1;
    int base, stride;
    line_base<DIM, N, S::LS>(dir, line, base, stride);
    base += el * S::NDP;
    // one metric per element: its row, loaded with the values of the test below
    // (after the vote it delayed the pairs: 32^3 p=4 FP32 179 -> 171 us)
    R met[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) met[d] = !NODAL && active ? sM[(el * DIM + dir) * DIM + d] : R(0);
    // straight-line pairs if every line of the warp's allows them
    bool straight = !active || ((!FASTABLE || !slow) && series_line<R, DIM, N, VOL, FS>(a.gas, sP, base, stride));
    straight = __all_sync(0xffffffffu, straight);
    if (active) {  // the barrier between the directions is every thread's
    const R *mrow = a.met + (long long)e * a.met_es + dir * DIM * a.met_cs;
    // NODAL: metric row of the line's node i
    auto row = [&](int i, R *m) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) m[d] = mrow[line_node<DIM, N>(dir, line, i) * a.met_ns + d * a.met_cs];
    };
    auto load = [&](int s, R *P) {
#pragma unroll
      for (int k = 0; k < PRIM; ++k) P[k] = sP[k * FS + s];
    };
    // averaged metric row of node j and a node with row mi (one row per
    // element: 0.5*(m+m) == m)
    auto pair_met = [&](const R *mi, int j, R *m) {
      if constexpr (NODAL) row(j, m);
#pragma unroll
      for (int d = 0; d < DIM; ++d) m[d] = NODAL ? R(0.5) * (mi[d] + m[d]) : mi[d];
    };
    if (straight) {
      // unrolled, the sums in registers: no branch separates the pairs, so
      // that several are in flight
      R acc[N][NEQ];
#pragma unroll
      for (int i = 0; i < N; ++i)
#pragma unroll
        for (int k = 0; k < NEQ; ++k) acc[i][k] = dir == 0 ? R(0) : sR[k * FS + base + i * stride];
#pragma unroll
      for (int i = 0; i < N - 1; ++i) {
        R A[PRIM];
        load(base + i * stride, A);
        if constexpr (NODAL) row(i, met);
#pragma unroll
        for (int j = i + 1; j < N; ++j) {
          R B[PRIM], m[DIM], F[NEQ];
          load(base + j * stride, B);
          pair_met(met, j, m);
          pair_flux<R, DIM, VOL, FASTABLE, LM_SERIES>(a.gas, A, B, m, F);
          const R ci = sD[i * N + j], cj = sD[j * N + i];
#pragma unroll
          for (int k = 0; k < NEQ; ++k) {
            acc[i][k] += ci * F[k];
            acc[j][k] += cj * F[k];
          }
        }
      }
#pragma unroll
      for (int i = 0; i < N; ++i)
#pragma unroll
        for (int k = 0; k < NEQ; ++k) sR[k * FS + base + i * stride] = acc[i][k];
    } else {
      // rolled, the sums in shared memory: the branches of the logarithmic
      // means, unrolled over the line, would outgrow the instruction cache
      if (dir == 0) {
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
          for (int k = 0; k < NEQ; ++k) sR[k * FS + base + i * stride] = R(0);
      }
#pragma unroll 1
      for (int i = 0; i < N - 1; ++i) {
        const int si = base + i * stride;
        R A[PRIM], sum[NEQ];
        load(si, A);
        if constexpr (NODAL) row(i, met);
#pragma unroll
        for (int k = 0; k < NEQ; ++k) sum[k] = sR[k * FS + si];
        auto pairs = [&](auto shared) {
#pragma unroll 1
          for (int j = i + 1; j < N; ++j) {
            const int sj = base + j * stride;
            R B[PRIM], m[DIM], F[NEQ];
            load(sj, B);
            pair_met(met, j, m);
            pair_flux<R, DIM, VOL, decltype(shared)::value, LM_BRANCH>(a.gas, A, B, m, F);
            const R ci = sD[i * N + j], cj = sD[j * N + i];
#pragma unroll
            for (int k = 0; k < NEQ; ++k) {
              sum[k] += ci * F[k];
              sR[k * FS + sj] += cj * F[k];
            }
          }
        };
        if (FASTABLE && slow) pairs(std::false_type{});  // outside the range of the shared reciprocals
        else pairs(std::integral_constant<bool, FASTABLE>{});
#pragma unroll
        for (int k = 0; k < NEQ; ++k) sR[k * FS + si] = sum[k];
      }
    }
#pragma unroll 1
    for (int i = 0; last && i < N; ++i) {
      R du[NEQ];
#pragma unroll
      for (int k = 0; k < NEQ; ++k) du[k] = sR[k * FS + base + i * stride];
      // node i of the column is summed
      const int n = line + i * NL;
      int f[DIM], fp[DIM];
      R w[DIM], fl[DIM][NEQ];
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        f[d] = d < DIM - 1 ? fd[d] : i == 0 ? fd[DIM - 1] : i == N - 1 ? fd[DIM] : -1;
        fp[d] = d == DIM - 1 ? line : DIM == 2 ? i : (d == 0 ? cy : cx) + N * i;
        // the lift's weights and fluxes: zero without a face, so that the
        // loads are predicated rather than branched around and issue together
        const bool in = lift_weight<R, DIM, S::NFP>(a, f[d], fp[d], w[d]);
#pragma unroll
        for (int k = 0; k < NEQ; ++k) {
          fl[d][k] = R(0);
          if (in) fl[d][k] = a.fstar[((long long)(f[d] >> 1) * NEQ + k) * S::NFP + fp[d]];
        }
      }
      if (i > 0 && a.jac_ns != 0) sc = R(1) / jac[(long long)i * NL * a.jac_ns];
      finish_node<R, DIM, N>(a, e, n, sc, al, dt, f, fp, w, fl, du, bad);
    }
    }
    if (!last) __syncthreads();
  }
  if (IsF32<R>::value && bad) atomicOr(a.status, STATUS_NONPOSITIVE);
}

// Threads of a line kernel whose CTAs hold EPB elements.
template <int DIM, int N, int EPB>
constexpr int line_threads() {
  return (EPB * (DIM == 2 ? N : N * N) + 31) / 32 * 32;
}

// Resident CTAs of T threads per SM that the registers are bounded for.  At
// 32^3 p=4 (N = 5), relative: FP64 three CTAs of 128 threads 1, four (spills)
// 1.06, two 1.16; FP32 five 1, six (spills) 1.01, four 1.04.  At 40^3 p=3
// (N = 4) FP64: four 1, three 1.01.  With a metric per node at p=5 (N = 6) the
// central flux spills at three: 16^3 Euler stage 254 us, 192 at two (the other
// fluxes, slower per pair: Ranocha 247 at three, 291 at two).
template <typename R, int N, int VOL, int T, bool NODAL = false>
constexpr int line_min_blocks() {
  return (IsF32<R>::value ? 5 : VOL == VOL_CENTRAL && N >= 6 && NODAL ? 2 : N >= 5 ? 3 : 4) * 128 / T;
}

template <typename R, int DIM, int N, int VOL, int T, bool NODAL>
__global__ void __launch_bounds__(T, (line_min_blocks<R, N, VOL, T, NODAL>())) volume_line_kernel(const VolArgs<R> a) {
  volume_line_body<R, DIM, N, VOL, T, 0, NODAL>(a, blockIdx.x);
}

}  // namespace thx
