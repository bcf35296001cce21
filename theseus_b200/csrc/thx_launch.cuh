// thx_launch.cuh -- typed launchers for the kernel templates and the names of
// the per-(precision, dimension, order) instantiation units.
#pragma once
#include "thx_kernels.cuh"
#include "thx_bc.cuh"

#include <algorithm>
#include <atomic>

namespace thx {

using PREC_T_0 = double;
using PREC_T_1 = float;

// Launch, with programmatic stream serialization (grid_start in the kernel)
// while the grid is small: there the launch latency is most of the time (RK3
// stage of the 32^2 p=3 vortex 9.8 -> 7.8 us).  CTAs of a large grid placed
// early take the SMs that the kernel before has left first, several on one,
// and the rest of the chip then waits for those (96^2 p=3 FP32-mixed 18.6 ->
// 27.1 us with the line kernel placed early).
constexpr unsigned kEarlyGrid = 5 * 148;
template <typename... P, typename... A>
cudaError_t launch_early(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A &&...args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = grid <= kEarlyGrid ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

template <typename R> using VolLaunch = cudaError_t (*)(const VolArgs<R> &, cudaStream_t, int prepare);
template <typename R> using FaceLaunch = cudaError_t (*)(const FaceArgs<R> &, cudaStream_t);
template <typename R> using GradLaunch = cudaError_t (*)(const GradArgs<R> &, cudaStream_t, int prepare);
template <typename R> using BlendLaunch = cudaError_t (*)(const BlendArgs<R> &, cudaStream_t);
// batched persistent forms: (argument table, work list, device work count,
// grid size, stream, prepare)
template <typename R>
using VolBatchLaunch = cudaError_t (*)(const VolArgs<R> *, const BatchWork *, const int *, int,
                                       cudaStream_t, int);
template <typename R>
using GradBatchLaunch = cudaError_t (*)(const GradArgs<R> *, const BatchWork *, const int *, int,
                                        cudaStream_t, int);
template <typename R>
using FaceBatchLaunch = cudaError_t (*)(const FaceArgs<R> *, const BatchWork *, const int *, int,
                                        cudaStream_t, int);

// The LTEEC volume kernel.
template <int DIM, int N, bool NS>
cudaError_t launch_volume_lte(const VolArgs<double> &a, cudaStream_t s, int prepare) {
  using S = Shape<DIM, N>;
  using M = LteVolSmem<DIM, N, NS>;
  if (prepare)
    return cudaFuncSetAttribute(volume_kernel_lte<DIM, N, NS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)M::bytes(true));
  if (a.ne <= 0) return cudaSuccess;
  return launch_early(volume_kernel_lte<DIM, N, NS>, (a.ne + S::EPB - 1) / S::EPB, S::THREADS, M::bytes(a.met_ns != 0),
                      s, a);
}

// The line kernel (ideal gas): one thread per tensor line.  NODAL: for meshes
// whose metric varies within the element.
template <typename R, int DIM, int N, int VOL, bool NODAL, int T = kLineThreads>
cudaError_t launch_volume_line(const VolArgs<R> &a, cudaStream_t s, int prepare) {
  using S = LineShape<DIM, N, T>;
  constexpr size_t smem = LineSmem<R, DIM, N, VOL, T, 0, NODAL>::bytes();
  if (prepare)
    return cudaFuncSetAttribute(volume_line_kernel<R, DIM, N, VOL, T, NODAL>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (a.ne <= 0) return cudaSuccess;
  volume_line_kernel<R, DIM, N, VOL, T, NODAL><<<(a.ne + S::EPB - 1) / S::EPB, T, smem, s>>>(a);
  return cudaGetLastError();
}

// Small meshes: volume and face terms in one launch (surf: the surface flux).
template <typename R>
using SmallLaunch = cudaError_t (*)(const VolArgs<R> &, const FaceArgs<R> &, int surf, cudaStream_t, int prepare);

template <typename R, int DIM, int N, int VOL, bool FACES>
cudaError_t launch_volume_small(const VolArgs<R> &a, const FaceArgs<R> &fa, int surf, cudaStream_t s, int prepare) {
  using M = SmallSmem<R, DIM, N, VOL, FACES>;
  const int epb = small_epb(DIM, N, a.ne, FACES, IsF32<R>::value);
  static_assert(M::bytes(small_epb(DIM, N, 1 << 30, FACES, IsF32<R>::value)) <= 200 * 1024, "shared memory");
  if (prepare)
    return cudaFuncSetAttribute(volume_small_kernel<R, DIM, N, VOL, FACES>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)M::bytes(small_epb(DIM, N, 1 << 30, FACES, IsF32<R>::value)));
  if (a.ne <= 0) return cudaSuccess;
  return launch_early(volume_small_kernel<R, DIM, N, VOL, FACES>, (a.ne + epb - 1) / epb, kSmallThreads, M::bytes(epb), s, a, fa, surf, epb);
}

// Persistent, bulk-copy-staged volume kernel (no blending): as many CTAs as
// fit on the device at once, each walking the element blocks.
template <typename R, int DIM, int N, int VOL>
cudaError_t launch_volume_tma(const VolArgs<R> &a, cudaStream_t s, int prepare) {
  using S = Shape<DIM, N>;
  using T_ = VolTmaSmem<R, DIM, N, VOL>;
  auto kern = volume_tma_kernel<R, DIM, N, VOL>;
  static int cap = 0;  // resident CTAs on the device
  if (prepare) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T_::bytes);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0, per = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, T_::T, T_::bytes)) != cudaSuccess) return e;
    cap = (per > 0 ? per : 1) * sms;
    return cudaSuccess;
  }
  if (a.ne <= 0) return cudaSuccess;
  const int nblocks = (a.ne + S::EPB - 1) / S::EPB;
  kern<<<std::min(nblocks, cap > 0 ? cap : 148), T_::T, T_::bytes, s>>>(a);
  return cudaGetLastError();
}

template <typename R, int DIM, int SURF, bool NS>
cudaError_t launch_face(const FaceArgs<R> &a, cudaStream_t s) {
  const int nfp = DIM == 2 ? a.N : a.N * a.N;
  const long long total = (long long)a.nf * nfp;
  if (total <= 0) return cudaSuccess;
  const int grid = (int)((total + 127) / 128);
  if constexpr (SURF == SURF_LTEEC) return launch_early(face_kernel_lte<DIM, NS>, grid, 128, 0, s, a);
  else if constexpr (IsF32<R>::value) return launch_early(face_kernel_f32<DIM, SURF, NS>, grid, 128, 0, s, a);
  else return launch_early(face_kernel_f64<DIM, SURF, NS>, grid, 128, 0, s, a);
}

template <typename R, int DIM, int N, bool LTE = false>
cudaError_t launch_grad(const GradArgs<R> &a, cudaStream_t s, int prepare) {
  using S = Shape<DIM, N>;
  constexpr size_t smem = grad_smem_bytes<R, DIM, N>();
  if constexpr (LTE) {
    if (prepare)
      return cudaFuncSetAttribute(grad_kernel_lte<DIM, N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem);
    if (a.ne <= 0) return cudaSuccess;
    return launch_early(grad_kernel_lte<DIM, N>, (a.ne + S::EPB - 1) / S::EPB, S::THREADS, smem, s, a);
  } else {
    if (prepare)
      return cudaFuncSetAttribute(grad_kernel<R, DIM, N, LTE>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (a.ne <= 0) return cudaSuccess;
    const int grid = (a.ne + S::EPB - 1) / S::EPB;
    return launch_early(grad_kernel<R, DIM, N, LTE>, grid, S::THREADS, smem, s, a);
  }
}

// Axis-aligned meshes: one thread per tensor line (ops: D and Dhat, on the
// host).  FP64 reads the precomputed entropy variables.
template <typename R>
using GradLineLaunch = cudaError_t (*)(const GradArgs<R> &, const double *D, const double *Dhat, cudaStream_t, int);

template <typename R, int DIM, int N>
cudaError_t launch_grad_line(const GradArgs<R> &a, const double *D, const double *Dhat, cudaStream_t s, int prepare) {
  constexpr int T = kLineThreads;
  constexpr bool SV = !IsF32<R>::value;
  using S = LineShape<DIM, N, T>;
  constexpr size_t smem = GradLineSmem<R, DIM, N, T>::bytes();
  if (prepare)
    return cudaFuncSetAttribute(grad_line_kernel<R, DIM, N, T, SV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem);
  if (a.ne <= 0) return cudaSuccess;
  if (SV && !a.svars) return cudaErrorInvalidValue;
  LineOps<R, N> m;
  for (int i = 0; i < N * N; ++i) {
    m.D[i] = (R)D[i];
    m.Dhat[i] = (R)Dhat[i];
  }
  grad_line_kernel<R, DIM, N, T, SV><<<(a.ne + S::EPB - 1) / S::EPB, T, smem, s>>>(a, m);
  return cudaGetLastError();
}

// Gradient from precomputed entropy variables (a.svars, entropy_kernel).
template <typename R, int DIM, int N>
cudaError_t launch_grad_sv(const GradArgs<R> &a, cudaStream_t s, int prepare) {
  using S = Shape<DIM, N>;
  constexpr size_t smem = grad_sv_smem_bytes<R, DIM, N>();
  if (prepare)
    return cudaFuncSetAttribute(grad_sv_kernel<R, DIM, N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem);
  if (a.ne <= 0) return cudaSuccess;
  if (!a.svars) return cudaErrorInvalidValue;
  const int grid = (a.ne + S::EPB - 1) / S::EPB;
  return launch_early(grad_sv_kernel<R, DIM, N>, grid, S::THREADS, smem, s, a);
}

template <typename R>
using EntropyLaunch = cudaError_t (*)(const R *, long long, const GasT<R> &, R *, cudaStream_t);

template <typename R, int DIM>
cudaError_t launch_entropy(const R *u, long long L, const GasT<R> &g, R *sv, cudaStream_t s) {
  if (L <= 0) return cudaSuccess;
  return launch_early(entropy_kernel<R, DIM>, (unsigned)((L + 255) / 256), 256, 0, s, u, L, g, sv);
}

template <int DIM>
cudaError_t launch_lte_temperature(const double *u, long long L, const LteDev &t, double *Tn,
                                   int *Cn, unsigned *status, cudaStream_t s) {
  if (L <= 0) return cudaSuccess;
  const int grid = (int)std::min<long long>((L + 255) / 256, 148LL * 8);
  return launch_early(lte_temperature_kernel<DIM>, grid, 256, 0, s, u, L, t, Tn, Cn, status);
}

// grid: in units of the CTAs that are resident at once on an SM; more than all
// of them balance the items better.
template <typename R, int DIM, int N, int VOL, bool NODAL, int T>
cudaError_t launch_volume_batched(const VolArgs<R> *args, const BatchWork *work, const int *nwork,
                                  int grid, cudaStream_t s, int prepare) {
  auto kern = volume_batched<R, DIM, N, VOL, NODAL, T>;
  constexpr size_t smem = LineSmem<R, DIM, N, VOL, T, 0, NODAL>::bytes();
  static std::atomic<int> resident{0};  // CTAs per SM
  if (prepare) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, T, smem);
    resident = per;
    return e;
  }
  if (grid <= 0) return cudaSuccess;
  kern<<<grid * std::max(1, resident.load()), T, smem, s>>>(args, work, nwork);
  return cudaGetLastError();
}

template <typename R, int DIM, int N, int VOL, int EPBX>
cudaError_t launch_volume_batched_pairs(const VolArgs<R> *args, const BatchWork *work, const int *nwork,
                                        int grid, cudaStream_t s, int prepare) {
  constexpr size_t smem = SmallSmem<R, DIM, N, VOL, false>::bytes(EPBX);
  if (prepare)
    return cudaFuncSetAttribute(volume_batched_pairs<R, DIM, N, VOL, EPBX>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (grid <= 0) return cudaSuccess;
  volume_batched_pairs<R, DIM, N, VOL, EPBX><<<grid, kSmallThreads, smem, s>>>(args, work, nwork);
  return cudaGetLastError();
}

template <typename R, int DIM, int N, int EPBX = 0>
cudaError_t launch_grad_batched(const GradArgs<R> *args, const BatchWork *work, const int *nwork,
                                int grid, cudaStream_t s, int prepare) {
  using S = Shape<DIM, N, EPBX>;
  constexpr size_t smem = grad_smem_bytes<R, DIM, N, EPBX>();
  if (prepare)
    return cudaFuncSetAttribute(grad_batched<R, DIM, N, EPBX>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (grid <= 0) return cudaSuccess;
  grad_batched<R, DIM, N, EPBX><<<grid, S::THREADS, smem, s>>>(args, work, nwork);
  return cudaGetLastError();
}

// Elements per CTA of the batched kernels' half-size variant (0: none, the
// full-size CTA already holds one element).
template <int DIM, int N>
constexpr int half_epb() {
  return Shape<DIM, N>::EPB >= 2 ? Shape<DIM, N>::EPB / 2 : 0;
}

template <typename R, int DIM, int SURF, bool NS>
cudaError_t launch_face_batched(const FaceArgs<R> *args, const BatchWork *work, const int *nwork,
                                int grid, cudaStream_t s, int prepare) {
  if (prepare || grid <= 0) return cudaSuccess;
  face_batched<R, DIM, SURF, NS><<<grid, 128, 0, s>>>(args, work, nwork);
  return cudaGetLastError();
}

// FP64 islands: walkers over device-side lists (grid fixed, length read on
// the device)
template <typename R>
using VolListLaunch = cudaError_t (*)(const VolArgs<R> &, const int *, const int *, cudaStream_t, int);
template <typename R>
using BlendListLaunch = cudaError_t (*)(const BlendArgs<R> &, const int *, const int *, cudaStream_t);
template <typename R>
using FaceListLaunch = cudaError_t (*)(const FaceArgs<R> &, const int *, cudaStream_t);
constexpr int kIslandGrid = 148 * 4;

template <typename R, int DIM, int N, int VOL, bool NODAL>
cudaError_t launch_volume_list(const VolArgs<R> &a, const int *list, const int *count, cudaStream_t s,
                               int prepare) {
  constexpr int T = line_list_threads<DIM, N>();
  constexpr size_t smem = LineSmem<R, DIM, N, VOL, T, Shape<DIM, N>::EPB, NODAL>::bytes();
  if (prepare)
    return cudaFuncSetAttribute(volume_list_kernel<R, DIM, N, VOL, NODAL>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  volume_list_kernel<R, DIM, N, VOL, NODAL><<<kIslandGrid, T, smem, s>>>(a, list, count);
  return cudaGetLastError();
}

template <typename R, int DIM, int N>
cudaError_t launch_fv_list(const VolArgs<R> &a, const int *list, const int *count, cudaStream_t s,
                           int prepare) {
  using S = Shape<DIM, N>;
  constexpr size_t smem = FvSmem<R, DIM, N>::bytes();
  if (prepare)
    return cudaFuncSetAttribute(fv_list_kernel<R, DIM, N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem);
  fv_list_kernel<R, DIM, N><<<kIslandGrid, S::THREADS, smem, s>>>(a, list, count);
  return cudaGetLastError();
}

template <typename R, int DIM, int N>
cudaError_t launch_blend_list(const BlendArgs<R> &a, const int *list, const int *count, cudaStream_t s) {
  return launch_early(blend_warp_kernel<R, DIM, N>, kIslandGrid, 32 * kBlendWarps, 0, s, a, list, count);
}

template <typename R, int DIM, int SURF>
cudaError_t launch_face_list(const FaceArgs<R> &a, const int *count, cudaStream_t s) {
  face_list_kernel<R, DIM, SURF><<<148 * 8, 128, 0, s>>>(a, count);
  return cudaGetLastError();
}

using BndLaunch = cudaError_t (*)(const BndArgs &, cudaStream_t);

template <int DIM, int SURF, bool NS>
cudaError_t launch_bnd(const BndArgs &a, cudaStream_t s) {
  const int nfp = DIM == 2 ? a.N : a.N * a.N;
  const long long total = (long long)a.nbf * nfp;
  if (total <= 0) return cudaSuccess;
  return launch_early(bnd_face_kernel<DIM, SURF, NS>, (unsigned)((total + 127) / 128), 128, 0, s, a);
}

template <typename R, int DIM, int N>
cudaError_t launch_fv(const VolArgs<R> &a, cudaStream_t s, int prepare) {
  using S = Shape<DIM, N>;
  constexpr size_t smem = FvSmem<R, DIM, N>::bytes();
  if (prepare)
    return cudaFuncSetAttribute(fv_kernel<R, DIM, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (a.ne <= 0 || !a.alpha || !a.fvrate) return cudaSuccess;
  const int grid = (a.ne + S::EPB - 1) / S::EPB;
  return launch_early(fv_kernel<R, DIM, N>, grid, S::THREADS, smem, s, a);
}

template <typename R, int DIM, int N>
cudaError_t launch_blend(const BlendArgs<R> &a, cudaStream_t s) {
  if (a.ne <= 0) return cudaSuccess;
  const int grid = (a.ne + kBlendWarps - 1) / kBlendWarps;  // one warp per element
  return launch_early(blend_warp_kernel<R, DIM, N>, grid, 32 * kBlendWarps, 0, s, a, nullptr, nullptr);
}

template <typename R>
struct OrderKernelsT {
  VolLaunch<R> vol[4][2];        // [volume flux][metric varies within the element]
  SmallLaunch<R> small[4][2];    // smaller meshes [volume flux][face terms too]
  VolLaunch<R> vol_tma[4];       // bulk-copy-staged
  GradLaunch<R> grad;
  GradLineLaunch<R> grad_line;   // axis-aligned meshes
  BlendLaunch<R> blend;
  VolLaunch<R> fv;               // subcell FV rate of blended elements
  VolBatchLaunch<R> volb[4][2];  // as vol
  GradBatchLaunch<R> gradb;
  // half-size CTAs (null when the gradient's full-size CTA holds one element)
  int epb, epb_half;             // elements per work item of the gradient kernels
  int vepb, vepb_half;           // of the volume kernels
  VolBatchLaunch<R> volb_half[4][2];
  GradBatchLaunch<R> gradb_half;
  // FP64 islands (Euler, blending; set in the FP64 units only)
  VolListLaunch<R> voll[4][2];   // as vol
  VolListLaunch<R> fvl;
  BlendListLaunch<R> blendl;
};
template <typename R>
struct FaceKernelsT {
  FaceLaunch<R> face[6][2];      // [surface flux][ns]
  FaceBatchLaunch<R> faceb[6][2];
  BndLaunch bnd[6][2];           // boundary faces [surface flux][ns] (FP64)
  EntropyLaunch<R> entropy;      // entropy variables of every node (NS)
  FaceListLaunch<R> facel[6];    // FP64 islands: listed faces (Euler; FP64 units only)
};
using OrderKernels0 = OrderKernelsT<double>;
using OrderKernels1 = OrderKernelsT<float>;
using FaceKernels0 = FaceKernelsT<double>;
using FaceKernels1 = FaceKernelsT<float>;
// LTE Helmholtz gas, FP64: LTEEC volume kernel [euler|ns], gradient, face
// flux [euler|ns].
struct LteKernels { VolLaunch<double> vol[2]; GradLaunch<double> grad; };
struct LteFaceKernels { FaceLaunch<double> face[2]; };

#define THX_DECLARE_ORDER(P, D, N) OrderKernels##P order_kernels_##P##_##D##_##N();
#define THX_DECLARE_FACE(P, D) FaceKernels##P face_kernels_##P##_##D();
#define THX_FOR_ORDERS(X, P, D) X(P, D, 3) X(P, D, 4) X(P, D, 5) X(P, D, 6)
THX_FOR_ORDERS(THX_DECLARE_ORDER, 0, 2)
THX_FOR_ORDERS(THX_DECLARE_ORDER, 0, 3)
THX_FOR_ORDERS(THX_DECLARE_ORDER, 1, 2)
THX_FOR_ORDERS(THX_DECLARE_ORDER, 1, 3)
#define THX_DECLARE_LTE(P, D, N) LteKernels lte_kernels_##D##_##N();
THX_FOR_ORDERS(THX_DECLARE_LTE, 0, 2)
THX_FOR_ORDERS(THX_DECLARE_LTE, 0, 3)
LteFaceKernels lte_face_kernels_2();
LteFaceKernels lte_face_kernels_3();
THX_DECLARE_FACE(0, 2)
THX_DECLARE_FACE(0, 3)
THX_DECLARE_FACE(1, 2)
THX_DECLARE_FACE(1, 3)

}  // namespace thx
