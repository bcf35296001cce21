// thx_grad.cuh -- BR1 gradient and viscous flux on axis-aligned meshes, one
// thread per tensor line (ideal gas).
//
// On a mesh whose elements are boxes along the axes (one metric per element,
// off-diagonal entries and off-axis normal components exactly zero) the
// gradient in direction d comes from the d-lines alone: derivative, metric and
// lift of a line's nodes are one thread's work, and the terms left out are
// products with zero.  The general kernels read every derivative term from
// shared memory once per node and stage nine lift factors per face point (75
// and up to 27 shared-memory reads per node, the shared-memory pipe 85 % busy);
// here a line's N values are read once per variable and the derivative matrix
// comes from the kernel's parameters.  Every sum keeps the general kernels'
// order, so the results are theirs.
#pragma once

namespace thx {

// Derivative matrix D and weak-form Dhat, in the parameter bank.
template <typename R, int N>
struct LineOps {
  R D[N * N], Dhat[N * N];
};

template <typename R, int DIM, int N, int T>
struct GradLineSmem {
  using S = LineShape<DIM, N, T>;
  static constexpr int FIELDS = DIM * S::NEQ;  // entropy variables, then the other directions' gradients
  static constexpr size_t bytes() {
    return sizeof(R) * (size_t)FIELDS * S::FS + sizeof(int) * 3 * S::EPB * 2 * DIM;
  }
};

// What the entropy variables at node i are formed from: themselves (SV:
// stored), or the working state, narrowed from the FP64 state as grad_body
// does where that is given.
template <typename R, int DIM, bool SV>
__device__ __forceinline__ void entropy_load(const GradArgs<R> &a, const long long L, const long long i, R *x) {
#pragma unroll
  for (int k = 0; k < DIM + 2; ++k) {
    if (SV) x[k] = a.svars[k * L + i];
    else x[k] = a.u64 ? (R)(a.u64[k * L + i] - a.off[k]) : a.u[k * L + i];
  }
}
template <typename R, int DIM, bool SV>
__device__ __forceinline__ void entropy_from(const GradArgs<R> &a, const R *x, R *w) {
  if constexpr (SV) {
#pragma unroll
    for (int k = 0; k < DIM + 2; ++k) w[k] = x[k];
  } else {
    R q[DIM + 2];
    reconstruct<R, DIM>(a.gas, x, q);
    entropy_vars<R, DIM>(a.gas, q, w);
  }
}

template <typename R, int DIM, int N, int T, bool SV>
__global__ void __launch_bounds__(T, IsF32<R>::value ? 5 : 3)
grad_line_kernel(const GradArgs<R> a, const LineOps<R, N> m) {
  using S = LineShape<DIM, N, T>;
  using M = GradLineSmem<R, DIM, N, T>;
  constexpr int ND = S::ND, NEQ = S::NEQ, NV = NEQ - 1, E = DIM + 1, EPB = S::EPB, NL = S::NL, FS = S::FS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (dynamic_smem_bytes() < M::bytes()) {
    if (threadIdx.x == 0 && a.status) atomicOr(a.status, STATUS_LAUNCH);
    return;
  }
  R *sS = reinterpret_cast<R *>(smem_raw);                     // [NEQ][EPB][NDP] entropy variables
  R *sG = sS + NEQ * FS;                                       // [DIM-1][NEQ][EPB][NDP] gradients
  int *sF = reinterpret_cast<int *>(sS + M::FIELDS * FS);      // [EPB][2*DIM] elem_face
  int *sNE = sF + EPB * 2 * DIM, *sNL = sNE + EPB * 2 * DIM;   // the neighbours' elements and local faces
  const int tid = threadIdx.x;
  const int e0 = blockIdx.x * EPB;
  const long long L = (long long)a.ne * ND;
  const int nodes = min(EPB, a.ne - e0) * ND;
  // every load of the thread's nodes is issued before the first use
  constexpr int IT = (EPB * ND + T - 1) / T;
  R xn[IT][NEQ];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int i = tid + it * T;
    if (i < nodes) entropy_load<R, DIM, SV>(a, L, (long long)e0 * ND + i, xn[it]);
  }
  for (int i = tid; i < nodes / ND * 2 * DIM; i += T) {
    const int fs = a.elem_face[(long long)e0 * 2 * DIM + i];
    const bool in = fs >= 0 && !(a.bw && (fs >> 1) >= a.nf_int);
    sF[i] = fs;
    sNE[i] = in ? a.face_elem[2 * (fs >> 1) + 1 - (fs & 1)] : 0;
    sNL[i] = in ? a.face_lface[2 * (fs >> 1) + 1 - (fs & 1)] : 0;
  }
  bool bad = false;
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int i = tid + it * T;
    if (i >= nodes) continue;
    R w[NEQ];
    if constexpr (IsF32<R>::value) {
      if (a.u64) {
        // the working copy of the node for the kernels that follow, and the
        // positivity of its FP64 state
        const long long gi = (long long)e0 * ND + i;
        double d[NEQ];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) d[k] = a.u64[k * L + gi];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) a.yf[k * L + gi] = (float)xn[it][k];
        if (!fp64_state_positive<DIM>(d, (double)a.gas.gm1)) bad = true;
      }
    }
    entropy_from<R, DIM, SV>(a, xn[it], w);
    const int pn = i + (N % 2 ? 0 : i / N);
#pragma unroll
    for (int k = 0; k < NEQ; ++k) sS[k * FS + pn] = w[k];
  }
  if (bad && a.status) atomicOr(a.status, STATUS_NONPOSITIVE);
  __syncthreads();

  const int el = tid / NL, line = tid - el * NL;
  const int e = e0 + el;
  const bool active = el < EPB && e < a.ne;
  const R *met = a.met + (long long)e * a.met_es;
  const R *jac = a.jac + (long long)e * a.jac_es;
  // the neighbours' traces, lift weights and normals at the ends of the
  // thread's lines: every gather is issued before the first derivative
  R so[DIM][2][NEQ], lw[DIM][2], ln[DIM][2];
  if (active) {
#pragma unroll
    for (int dir = 0; dir < DIM; ++dir)
#pragma unroll
      for (int hi = 0; hi < 2; ++hi) {
        const int lf = el * 2 * DIM + 2 * dir + hi, fs = sF[lf], f = fs >> 1;
        if (fs < 0 || (a.bw && f >= a.nf_int)) continue;
        entropy_load<R, DIM, SV>(a, L, (long long)sNE[lf] * ND + trace_node<DIM>(N, sNL[lf], line), so[dir][hi]);
        lw[dir][hi] = ((fs & 1) == 0 ? a.wm : a.wp)[(long long)f * a.w_fs + (long long)line * a.w_ps];
        ln[dir][hi] = a.normal[((long long)f * a.n_fs + (long long)line * a.n_ps) * DIM + dir];
      }
  }
  // gradient along `dir` of the thread's line: invJ * (D-derivative * metric)
  // plus the lift of the end nodes' faces
  auto gradient = [&](auto dirc, R *dst) {
    constexpr int dir = decltype(dirc)::value;
    int base, stride;
    line_base<DIM, N, S::LS>(dir, line, base, stride);
    base += el * S::NDP;
    R lift[2][NEQ];
    bool lifted[2];
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      const int fs = sF[el * 2 * DIM + 2 * dir + hi];
      const int f = fs >> 1, side = fs & 1;
      const int own = base + (hi ? N - 1 : 0) * stride;
      lifted[hi] = fs >= 0;
#pragma unroll
      for (int k = 0; k < NEQ; ++k) lift[hi][k] = R(0);
      if (fs < 0) continue;
      if constexpr (!IsF32<R>::value) {
        if (a.bw && f >= a.nf_int) {
          // boundary face (include/NSOperator_impl.hpp:285-404): w_b (exterior
          // - interior entropy variables) n
          const int b = f - a.nf_int;
          const long long bp = (long long)b * S::NFP + line;
          R w[NEQ], fl[NEQ];
#pragma unroll
          for (int k = 0; k < NEQ; ++k) w[k] = sS[k * FS + own];
          bc_grad_flux<DIM>(a.gas, a.bcs[a.bdr_bc[b]], a.bc_data, w, fl);
          const R scale = a.bw[bp], n = a.bnrm[bp * DIM + dir];
#pragma unroll
          for (int k = 0; k < NEQ; ++k) lift[hi][k] += scale * (fl[k] * n);
          continue;
        }
      }
      // interior face: w * 0.5 (S+ - S-) n
      R st[NEQ];
      entropy_from<R, DIM, SV>(a, so[dir][hi], st);
#pragma unroll
      for (int k = 0; k < NEQ; ++k) {
        const R sown = sS[k * FS + own];
        const R jump = side == 0 ? R(0.5) * (st[k] - sown) : R(0.5) * (sown - st[k]);
        lift[hi][k] += lw[dir][hi] * (jump * ln[dir][hi]);
      }
    }
    const R ar = met[dir * DIM + dir];
    R ij[N];
#pragma unroll
    for (int i = 0; i < N; ++i)
      ij[i] = i > 0 && a.jac_ns == 0 ? ij[0] : R(1) / jac[(long long)line_node<DIM, N>(dir, line, i) * a.jac_ns];
    // rolled over the variables: unrolled, the kernel outgrows the
    // instruction cache
#pragma unroll 1
    for (int k = 0; k < NEQ; ++k) {
      R s[N];
#pragma unroll
      for (int l = 0; l < N; ++l) s[l] = sS[k * FS + base + l * stride];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        R g = R(0);
#pragma unroll
        for (int l = 0; l < N; ++l) g += s[l] * m.D[i * N + l];
        g = g * ar;
        dst[k * FS + base + i * stride] = ij[i] * g;
      }
    }
#pragma unroll
    for (int hi = 0; hi < 2; ++hi)
      if (lifted[hi]) {
#pragma unroll
        for (int k = 0; k < NEQ; ++k) dst[k * FS + base + (hi ? N - 1 : 0) * stride] += lift[hi][k];
      }
  };
  if (active) {
    gradient(std::integral_constant<int, 0>{}, sG);
    if constexpr (DIM == 3) gradient(std::integral_constant<int, 1>{}, sG + NEQ * FS);
  }
  __syncthreads();
  // The last direction's gradient replaces the column's entropy variables;
  // then, node by node, the gradients become primitive gradients and the
  // physical viscous flux (include/NavierStokesFlux.hpp:160-290), whose
  // contravariant components take the gradients' places.
  if (active) {
    gradient(std::integral_constant<int, DIM - 1>{}, sS);
    int base, stride;
    line_base<DIM, N, S::LS>(DIM - 1, line, base, stride);
    base += el * S::NDP;
    R row[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) row[d] = met[d * DIM + d];
    // the next node's state is loaded while this one's flux is formed
    R next[NEQ];
    auto fetch = [&](int i) {
      const long long gi = (long long)e * ND + line + i * NL;
#pragma unroll
      for (int k = 0; k < NEQ; ++k) {
        if (!SV && a.u64) next[k] = (R)(a.u64[k * L + gi] - a.off[k]);
        else next[k] = a.u[k * L + gi];
      }
    };
    fetch(0);
#pragma unroll 1
    for (int i = 0; i < N; ++i) {
      const int s = base + i * stride, n = line + i * NL;
      const long long gi = (long long)e * ND + n;
      R q[NEQ], g[DIM][NEQ];
      reconstruct<R, DIM>(a.gas, next, q);
      if (i + 1 < N) fetch(i + 1);
      const NodeGas<R, DIM> ng = node_gas<R, DIM>(a.gas, q);
#pragma unroll
      for (int cc = 0; cc < DIM; ++cc) {
        R ge[NEQ];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) ge[k] = (cc == DIM - 1 ? sS : sG + cc * NEQ * FS)[k * FS + s];
        grad_entropy_to_prim_ng<R, DIM>(ng, q, ge, g[cc]);
      }
      const R mu = viscosity_ng<R, DIM>(a.gas, ng);
      const R kappa = mu * a.gas.cp * a.gas.Pr_inv;
      const R fac = fdiv(a.gas.gm1_inv, a.gas.cv * ng.rho);
      R div = R(0);
#pragma unroll
      for (int d = 0; d < DIM; ++d) div += g[d][1 + d];
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        R ef = kappa * (fac * (g[d][E] - ng.p_rho * g[d][0]));
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
          R tau;
          if (c == d) tau = mu * (R(2) * g[d][1 + c] - a.gas.mu_bulk * div);
          else tau = mu * (g[d][1 + c] + g[c][1 + d]);
          a.vflux[((long long)d * NV + c) * L + gi] = tau;
          sS[(d * NV + c) * FS + s] = row[d] * tau;
          ef += ng.v[c] * tau;
        }
        a.vflux[((long long)d * NV + DIM) * L + gi] = ef;
        sS[(d * NV + DIM) * FS + s] = row[d] * ef;
      }
      // primitive gradients at this node's boundary points, for the viscous
      // boundary fluxes
      if constexpr (!IsF32<R>::value) {
        if (a.bw) {
          int c[3];
          node_coords<DIM, N>(n, c);
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            if (c[d] != 0 && c[d] != N - 1) continue;
            const int fs = sF[el * 2 * DIM + 2 * d + (c[d] == N - 1 ? 1 : 0)];
            if (fs < 0 || (fs >> 1) < a.nf_int) continue;
            const long long bp = (long long)((fs >> 1) - a.nf_int) * S::NFP + face_point<DIM, N>(d, c);
#pragma unroll
            for (int k = 0; k < DIM * NEQ; ++k) a.bgrad[bp * DIM * NEQ + k] = (&g[0][0])[k];
          }
        }
      }
    }
  }
  // weak-form divergence with Dhat (include/DGSEMIntegrator.hpp:526-622): the
  // directions continue one another's sums, which take the places of the
  // contravariant components just read
#pragma unroll
  for (int dir = 0; dir < DIM; ++dir) {
    __syncthreads();
    if (!active) continue;
    int base, stride;
    line_base<DIM, N, S::LS>(dir, line, base, stride);
    base += el * S::NDP;
#pragma unroll 1
    for (int k = 0; k < NV; ++k) {
      R f[N];
#pragma unroll
      for (int l = 0; l < N; ++l) f[l] = sS[(dir * NV + k) * FS + base + l * stride];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        R dv = dir == 0 ? R(0) : sS[((dir - 1) * NV + k) * FS + base + i * stride];
#pragma unroll
        for (int l = 0; l < N; ++l) dv += m.Dhat[i * N + l] * f[l];
        if (dir < DIM - 1) sS[(dir * NV + k) * FS + base + i * stride] = dv;
        else a.vdiv[k * L + (long long)e * ND + line + i * NL] = dv;
      }
    }
  }
}

}  // namespace thx
