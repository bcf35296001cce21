// thx_inst_order.cu -- instantiates the volume, gradient and indicator kernels
// of one (precision, dimension, order) triple.  Compiled once per triple with
// -DTHX_PREC=<0 double|1 float> -DTHX_DIM=<2|3> -DTHX_N=<nodes per direction>.
#include "thx_launch.cuh"

#ifndef THX_PREC
#error "THX_PREC must be defined"
#endif

#define THX_CAT4(a, b, c, d) a##_##b##_##c##_##d
#define THX_NAME(P, D, N) THX_CAT4(order_kernels, P, D, N)
#define THX_TYPE2(P) OrderKernels##P
#define THX_TYPE(P) THX_TYPE2(P)
#define THX_RT2(P) PREC_T_##P
#define THX_RT(P) THX_RT2(P)

namespace thx {

THX_TYPE(THX_PREC) THX_NAME(THX_PREC, THX_DIM, THX_N)() {
  using R = THX_RT(THX_PREC);
  THX_TYPE(THX_PREC) k;
#define THX_SETV(V)                                           \
  k.vol[V][0] = &launch_volume_line<R, THX_DIM, THX_N, V, false>; \
  k.vol[V][1] = &launch_volume_line<R, THX_DIM, THX_N, V, true>;  \
  k.small[V][0] = &launch_volume_small<R, THX_DIM, THX_N, V, false>; \
  k.small[V][1] = &launch_volume_small<R, THX_DIM, THX_N, V, true>;  \
  k.vol_tma[V] = &launch_volume_tma<R, THX_DIM, THX_N, V>;     \
  k.volb[V][0] = &launch_volume_batched<R, THX_DIM, THX_N, V, false, batch_threads<R, THX_DIM, THX_N>()>; \
  k.volb[V][1] = &launch_volume_batched<R, THX_DIM, THX_N, V, true, batch_threads<R, THX_DIM, THX_N>()>;
  THX_SETV(VOL_CHANDRASHEKAR)
  THX_SETV(VOL_RANOCHA)
  THX_SETV(VOL_PIROZZOLI)
  THX_SETV(VOL_CENTRAL)
#undef THX_SETV
#if THX_PREC == 0
  k.grad = &launch_grad_sv<R, THX_DIM, THX_N>;  // FP64: entropy variables precomputed
#else
  k.grad = &launch_grad<R, THX_DIM, THX_N>;     // FP32: evaluated in the kernel (cheaper)
#endif
  k.grad_line = &launch_grad_line<R, THX_DIM, THX_N>;
  k.blend = &launch_blend<R, THX_DIM, THX_N>;
  k.fv = &launch_fv<R, THX_DIM, THX_N>;
  k.gradb = &launch_grad_batched<R, THX_DIM, THX_N>;
  k.epb = Shape<THX_DIM, THX_N>::EPB;
  k.epb_half = half_epb<THX_DIM, THX_N>();
  k.vepb = LineShape<THX_DIM, THX_N, batch_threads<R, THX_DIM, THX_N>()>::EPB;
  k.vepb_half = k.epb_half;
  for (auto &row : k.volb_half)
    for (auto &v : row) v = nullptr;
  k.gradb_half = nullptr;
  if constexpr (half_epb<THX_DIM, THX_N>() > 0) {
    constexpr int H = half_epb<THX_DIM, THX_N>();
    // FP64: the line and the pair kernel give the same bits
#if THX_PREC == 0
#define THX_SETH(V) k.volb_half[V][0] = k.volb_half[V][1] = &launch_volume_batched_pairs<R, THX_DIM, THX_N, V, H>;
#else
    k.vepb_half = k.vepb;
#define THX_SETH(V)                      \
  k.volb_half[V][0] = k.volb[V][0];      \
  k.volb_half[V][1] = k.volb[V][1];
#endif
    THX_SETH(VOL_CHANDRASHEKAR)
    THX_SETH(VOL_RANOCHA)
    THX_SETH(VOL_PIROZZOLI)
    THX_SETH(VOL_CENTRAL)
#undef THX_SETH
    k.gradb_half = &launch_grad_batched<R, THX_DIM, THX_N, H>;
  }
#if THX_PREC == 0
#define THX_SETL(V)                                                  \
  k.voll[V][0] = &launch_volume_list<R, THX_DIM, THX_N, V, false>; \
  k.voll[V][1] = &launch_volume_list<R, THX_DIM, THX_N, V, true>;
  THX_SETL(VOL_CHANDRASHEKAR)
  THX_SETL(VOL_RANOCHA)
  THX_SETL(VOL_PIROZZOLI)
  THX_SETL(VOL_CENTRAL)
#undef THX_SETL
  k.fvl = &launch_fv_list<R, THX_DIM, THX_N>;
  k.blendl = &launch_blend_list<R, THX_DIM, THX_N>;
#else
  for (auto &row : k.voll)
    for (auto &v : row) v = nullptr;
  k.fvl = nullptr;
  k.blendl = nullptr;
#endif
  return k;
}

}  // namespace thx
