// thx_small.cuh -- volume and face terms of a small mesh (ideal gas) in one
// kernel.
//
// What bounds a mesh of a few elements per SM is latency: the launches, the
// trips to memory and the longest chain of arithmetic in a thread.  So one
// launch does the face and the volume kernel's work (each element evaluates
// its own faces' fluxes, twice the flops, no trip through memory), the
// elements are spread over all SMs (a few per CTA, chosen at launch), the
// pairs of all directions are evaluated at once, one or two per thread, and
// two barriers separate node data and face fluxes, pair fluxes, and sums.
#pragma once

namespace thx {

constexpr int kSmallThreads = 256;
constexpr int kSmallSMs = 148;

// Elements per CTA.  With the face terms: spread over the SMs, up to about two
// pairs per thread.  Without: over three CTAs per SM in FP64 and four in FP32
// (see small_mesh), up to a node per thread.
__host__ constexpr int small_epb(int dim, int N, int ne, bool faces, bool f32) {
  const int nd = dim == 2 ? N * N : N * N * N;
  const int pairs = dim * (nd / N) * (N * (N - 1) / 2);
  const int most = faces ? 2 * kSmallThreads / pairs : kSmallThreads / nd;
  const int ctas = faces ? kSmallSMs : (f32 ? 4 : 3) * kSmallSMs;
  const int spread = (ne + ctas - 1) / ctas;
  const int epb = spread < most ? spread : most;
  return epb > 1 ? epb : 1;
}

// Which volume kernel a mesh takes: 2 this one with the face terms, 1 this one
// after the face kernel, 0 the line kernel after the face kernel.  The first
// two up to two, and three or four, CTAs per SM, which their registers allow at
// once; beyond, the line kernel's fewer instructions outweigh its longer chains.
// RK3 stage, Euler FP64, first / second / line kernel: 2-D p=3 32^2 7.6 / 9.8 /
// 19.0 us, 48^2 8.8 / 10.8 / 17.6, 64^2 14.8 / 13.9 / 18.3, 96^2 27.1 / 19.6 /
// 21.0, 128^2 41.2 / 30.7 / 28.4; 3-D p=3 5^3 8.6 / 11.7 / 25.2, 7^3 15.5 / 13.5 /
// 26.9, 16^3 103 / 52 / 50.  Shared memory holds only two FP64 CTAs of the second
// per SM at 3-D p=5, and at 3-D p=4 with all fluxes but Ranocha's: the last of
// three then run in a second wave, with which the kernel still beats the line
// kernel (p=5 441 elements 35.6 / 46.9 us Ranocha; p=4 840 elements 28.6 / 41.4
// Chandrashekar), except with the central flux (27.1 / 22.9, 25.3 / 23.0).
__host__ constexpr int small_mesh(int dim, int N, int ne, bool f32) {
  const int e2 = small_epb(dim, N, ne, true, f32), e1 = small_epb(dim, N, ne, false, f32);
  return (ne + e2 - 1) / e2 <= 2 * kSmallSMs ? 2 : (ne + e1 - 1) / e1 <= (f32 ? 4 : 3) * kSmallSMs ? 1 : 0;
}

template <typename R, int DIM, int N, int VOL, bool FACES>
struct SmallSmem {
  using S = Shape<DIM, N>;
  static constexpr int PRIM = node_fields<R, DIM, VOL>();
  static constexpr int FP = S::NEQ % 2 ? S::NEQ : S::NEQ + 1;  // stride of a pair's flux (odd: banks)
  static constexpr int PT = (DIM * S::PAIRS * 4 + 7) / 8 * 8;  // bytes of the pair table
  // values of R per element
  static constexpr int ELEM = PRIM * S::ND + DIM * S::PAIRS * FP +
                              (FACES ? 2 * DIM * S::NEQ * S::NFP : 0);
  __host__ __device__ static constexpr size_t bytes(int epb) {
    return PT + sizeof(R) * (size_t)(S::OPS + epb * ELEM) + sizeof(int) * (size_t)epb * 2 * DIM;
  }
};

// The work of elements [e0, e0 + epb).  FACES: the kernel evaluates the face
// fluxes itself; otherwise the face kernel has stored them.  EARLY: the kernel
// may have been launched early (grid_wait).
template <typename R, int DIM, int N, int VOL, bool FACES, bool EARLY>
__device__ __forceinline__ void small_body(const VolArgs<R> &a, const FaceArgs<R> &fa, const int surf, const int epb,
                                           const int e0) {
  using S = Shape<DIM, N>;
  using M = SmallSmem<R, DIM, N, VOL, FACES>;
  constexpr int ND = S::ND, NEQ = S::NEQ, NFP = S::NFP, PAIRS = S::PAIRS, PRIM = M::PRIM, T = kSmallThreads;
  constexpr bool FASTABLE = !IsF32<R>::value && (VOL == VOL_CHANDRASHEKAR || VOL == VOL_RANOCHA);
  if (EARLY) grid_release();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (dynamic_smem_bytes() < M::bytes(epb)) {
    if (threadIdx.x == 0) atomicOr(a.status, STATUS_LAUNCH);
    return;
  }
  unsigned *sPT = reinterpret_cast<unsigned *>(smem_raw);  // [DIM][PAIRS] lower node | upper << 16
  R *sD = reinterpret_cast<R *>(smem_raw + M::PT);         // Dhat2
  R *sP = sD + S::OPS;                                     // [epb][PRIM][ND]
  R *sB = sP + epb * PRIM * ND;                            // [epb][DIM][PAIRS][FP] pair fluxes
  R *sF = sB + epb * DIM * PAIRS * M::FP;                  // [epb][2*DIM][NEQ][NFP] face fluxes
  int *sE = reinterpret_cast<int *>(sF + (FACES ? epb * 2 * DIM * NEQ * NFP : 0));  // [epb][2*DIM] elem_face
  const int tid = threadIdx.x;
  const int cnt = min(epb, a.ne - e0);
  const long long L = (long long)a.ne * ND;
  for (int i = tid; i < N * N; i += T) sD[i] = a.ops[i];
  for (int i = tid; i < DIM * PAIRS; i += T) {
    const int dir = i / PAIRS, p = i % PAIRS;
    int lo, hi;
    pair_decode<N>(p % S::NP, lo, hi);
    const int line = p / S::NP;
    sPT[i] = (unsigned)line_node<DIM, N>(dir, line, lo) | ((unsigned)line_node<DIM, N>(dir, line, hi) << 16);
  }
  if (EARLY) grid_wait();  // what precedes reads the mesh only
  if (!FACES)
    for (int i = tid; i < cnt * 2 * DIM; i += T) sE[i] = a.elem_face[(long long)e0 * 2 * DIM + i];
  // face fluxes; a boundary face's is the boundary kernel's
  for (int t = tid; FACES && t < cnt * 2 * DIM * NFP; t += T) {
    const int ef = t / NFP, fp = t - ef * NFP;
    const int fs = a.elem_face[(long long)e0 * 2 * DIM + ef];
    if (fp == 0) sE[ef] = fs;
    if (fs < 0) continue;
    const int f = fs >> 1;
    if (!IsF32<R>::value && a.bw && f >= a.nf_int) continue;
    R F[NEQ];
    if (fa.vflux) face_point_flux<R, DIM, -1, true>(fa, f, fp, F, surf);
    else face_point_flux<R, DIM, -1, false>(fa, f, fp, F, surf);
#pragma unroll
    for (int k = 0; k < NEQ; ++k) sF[(ef * NEQ + k) * NFP + fp] = F[k];
  }
  // node data
  bool slow = false;
  for (int i = tid; i < cnt * ND; i += T) {
    const int el = i / ND, n = i - el * ND;
    R q[NEQ], pr[nprim<R, DIM>()], fl[PRIM];
#pragma unroll
    for (int k = 0; k < NEQ; ++k) q[k] = a.u[k * L + (long long)e0 * ND + i];
    node_prims<R, DIM, VOL>(a.gas, q, pr);
    pack_node<R, DIM, VOL>(a.gas, q, pr, fl);
#pragma unroll
    for (int k = 0; k < PRIM; ++k) sP[(el * PRIM + k) * ND + n] = fl[k];
    if constexpr (!IsF32<R>::value) {
      if (!(pr[0] > R(0)) || !(pr[DIM + 1] > R(0))) atomicOr(a.status, STATUS_NONPOSITIVE);
      if constexpr (FASTABLE) slow = slow || !in_fast_range(pr[0]) || !in_fast_range(pr[DIM + 1]);
    }
  }
  if constexpr (FASTABLE) slow = __syncthreads_or(slow);
  else __syncthreads();
  // every symmetric pair of every direction once, in (lower, upper) order
  for (int t = tid; t < cnt * DIM * PAIRS; t += T) {
    const int el = t / (DIM * PAIRS), p = t - el * (DIM * PAIRS), dir = p / PAIRS;
    const int na = (int)(sPT[p] & 0xffffu), nb = (int)(sPT[p] >> 16);
    R A[PRIM], B[PRIM], met[DIM], F[NEQ];
#pragma unroll
    for (int k = 0; k < PRIM; ++k) {
      A[k] = sP[(el * PRIM + k) * ND + na];
      B[k] = sP[(el * PRIM + k) * ND + nb];
    }
    // one metric row per element: 0.5*(m+m) == m
    const R *m = a.met + (long long)(e0 + el) * a.met_es + dir * DIM * a.met_cs;
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      met[d] = a.met_ns == 0 ? m[d] : R(0.5) * (m[na * a.met_ns + d * a.met_cs] + m[nb * a.met_ns + d * a.met_cs]);
    if (FASTABLE && slow) pair_flux<R, DIM, VOL, false, LM_BRANCH>(a.gas, A, B, met, F);
    else pair_flux<R, DIM, VOL, FASTABLE, LM_BRANCH>(a.gas, A, B, met, F);
#pragma unroll
    for (int k = 0; k < NEQ; ++k) sB[t * M::FP + k] = F[k];
  }
  __syncthreads();
  // rate_i = sum over directions and m of Dhat2(i,m) F(i,m), in that order
  const double dt = a.stage == 0 ? 0.0 : a.dt_dev ? *a.dt_dev : a.dt;
  bool bad = false;
  for (int i = tid; i < cnt * ND; i += T) {
    const int el = i / ND, n = i - el * ND, e = e0 + el;
    int c[3];
    node_coords<DIM, N>(n, c);
    R du[NEQ], w[DIM], fl[DIM][NEQ];
    int f[DIM], fp[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const bool edge = c[d] == 0 || c[d] == N - 1;
      const int ef = el * 2 * DIM + 2 * d + (c[d] == N - 1 ? 1 : 0);
      f[d] = edge ? sE[ef] : -1;
      fp[d] = face_point<DIM, N>(d, c);
      const bool in = lift_weight<R, DIM, NFP>(a, f[d], fp[d], w[d]);
#pragma unroll
      for (int k = 0; k < NEQ; ++k) {
        fl[d][k] = R(0);
        if (in) fl[d][k] = FACES ? sF[(ef * NEQ + k) * NFP + fp[d]] : a.fstar[((long long)(f[d] >> 1) * NEQ + k) * NFP + fp[d]];
      }
    }
#pragma unroll
    for (int k = 0; k < NEQ; ++k) du[k] = R(0);
#pragma unroll
    for (int dir = 0; dir < DIM; ++dir) {
      const int me = c[dir], line = line_of<DIM, N>(dir, c);
#pragma unroll
      for (int m = 0; m < N; ++m) {
        if (m == me) continue;
        const int lo = m < me ? m : me, hi = m < me ? me : m;
        const R *F = sB + ((el * DIM + dir) * PAIRS + line * S::NP + pair_index<N>(lo, hi)) * M::FP;
        const R co = sD[me * N + m];
#pragma unroll
        for (int k = 0; k < NEQ; ++k) du[k] += co * F[k];
      }
    }
    const R sc = R(1) / a.jac[(long long)e * a.jac_es + (long long)n * a.jac_ns];
    finish_node<R, DIM, N>(a, e, n, sc, a.alpha ? a.alpha[e] : 0.0, dt, f, fp, w, fl, du, bad);
  }
  if (IsF32<R>::value && bad) atomicOr(a.status, STATUS_NONPOSITIVE);
}

template <typename R, bool FACES>
constexpr int small_min_blocks() {
  return FACES ? 2 : (IsF32<R>::value ? 4 : 3);
}

template <typename R, int DIM, int N, int VOL, bool FACES>
__global__ void __launch_bounds__(kSmallThreads, (small_min_blocks<R, FACES>()))
volume_small_kernel(const VolArgs<R> a, const FaceArgs<R> fa, const int surf, const int epb) {
  small_body<R, DIM, N, VOL, FACES, true>(a, fa, surf, epb, blockIdx.x * epb);
}

}  // namespace thx
