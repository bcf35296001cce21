// Device check of the shared reciprocals (theseus_b200/csrc/thx_volume.cuh and
// thx_face.cuh) against CUDA's own division: reciprocals within their bounds;
// quotients, logarithmic means, pair fluxes, entropy variables and surface
// fluxes equal to the separately divided forms of thx_device.cuh.  Prints one
// line per check: name, failures, samples.  Writes (x, log_normal(x), log(x))
// to the file argv[1].  Built with --fmad=false, as the library's FP64 units.
#include "thx_kernels.cuh"

#include <cstdio>

using namespace thx;

constexpr int kChecks = 12;
static const char *const kNames[kChecks] = {
    "rcp_refined", "div_by", "log_means", "log_means_reciprocals", "log_means_series", "pair_chandrashekar",
    "pair_ranocha", "entropy_vars", "surface_chandrashekar", "surface_hll", "surface_llf", "surface_roe"};
constexpr int kBlock = 128, kGrid = 148 * 32, kPer = 32;

struct Rng {
  unsigned long long s;
  __device__ unsigned long long next() {
    unsigned long long z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  }
  __device__ double uniform(double lo, double hi) { return lo + (hi - lo) * ((double)(next() >> 11) * 0x1p-53); }
  // mantissa in [1, 2), exponent in [-e, e); one in 64 at each end of the
  // range.  (Random significands there too: a power of two over a significand of
  // all ones lies 2^-53 ulp from a rounding boundary, closer than div_by
  // resolves, and round values would make such pairs often.)
  __device__ double scaled(int e) {
    const unsigned r = next() & 63;
    if (r == 0) return ldexp(1.0 + uniform(0.0, 0x1p-20), -e);
    if (r == 1) return ldexp(2.0 - uniform(0x1p-30, 0x1p-20), e - 1);
    return ldexp(uniform(1.0, 2.0), (int)(next() % (2 * e)) - e);
  }
  // a partner of x: equal, nearly equal, at the branch of the logarithmic
  // mean (ratio 1.02020...), or anywhere in the range
  __device__ double partner(double x, int e) {
    double y;
    switch (next() & 7) {
      case 0: return x;
      case 1: y = x * (1.0 + ldexp(uniform(-1.0, 1.0), -(int)(next() % 50))); break;
      case 2: y = x * (1.0202020202020203 * (1.0 + ldexp(uniform(-1.0, 1.0), -20 - (int)(next() % 32)))); break;
      case 3: y = x / (1.0202020202020203 * (1.0 + ldexp(uniform(-1.0, 1.0), -20 - (int)(next() % 32)))); break;
      case 4:
      case 5: y = x * uniform(0.5, 2.0); break;
      default: y = scaled(e); break;
    }
    return y >= ldexp(1.0, -e) && y < ldexp(1.0, e) ? y : scaled(e);
  }
};

__device__ bool same(double a, double b) { return a == b || (a != a && b != b); }
// |a - b| in units of b's last place
__device__ double ulps(double a, double b) {
  return fabs(a - b) / ldexp(1.0, ilogb(b) - 52);
}

// A gas state whose density and pressure lie within 2^-e .. 2^e.
template <int DIM>
__device__ void state(Rng &r, const GasT<double> &g, double rho, double p, double *q) {
  double m2 = 0.0;
  // speeds up to a few times that of sound; some exactly zero
  const double c = sqrt(p / rho);
  for (int d = 0; d < DIM; ++d) {
    q[1 + d] = (r.next() & 7) ? rho * c * r.uniform(-3.0, 3.0) : 0.0;
    m2 += q[1 + d] * q[1 + d];
  }
  q[0] = rho;
  q[DIM + 1] = p / g.gm1 + 0.5 * m2 / rho;
}

template <int DIM>
__device__ void fluxes(Rng &r, const GasT<double> &g, unsigned long long *bad) {
  constexpr int NEQ = DIM + 2;
  const int e = (r.next() & 1) ? 99 : 4;
  const double rho1 = r.scaled(e), p1 = r.scaled(e), rho2 = r.partner(rho1, e), p2 = r.partner(p1, e);
  double q1[NEQ], q2[NEQ], a[DIM + 3], b[DIM + 3], n[DIM], F[NEQ], G[NEQ];
  state<DIM>(r, g, rho1, p1, q1);
  state<DIM>(r, g, rho2, p2, q2);
  for (int d = 0; d < DIM; ++d) n[d] = r.uniform(-1.0, 1.0);
  auto differ = [&]() {
    for (int k = 0; k < NEQ; ++k)
      if (!same(F[k], G[k])) return true;
    return false;
  };
  node_prims<double, DIM, VOL_CHANDRASHEKAR>(g, q1, a);
  node_prims<double, DIM, VOL_CHANDRASHEKAR>(g, q2, b);
  if (in_fast_range(a[0]) && in_fast_range(b[0]) && in_fast_range(a[DIM + 1]) && in_fast_range(b[DIM + 1])) {
    vol_chandrashekar<double, DIM>(g, a, b, n, F);
    pair_chandrashekar<DIM, LM_BRANCH>(g, a, b, n, G);
    if (differ()) ++bad[5];
    vol_ranocha<double, DIM>(g, a, b, n, F);
    pair_ranocha<DIM, LM_BRANCH>(g, a, b, n, G);
    if (differ()) ++bad[6];
  }
  entropy_vars<double, DIM>(g, q1, F);
  entropy_vars_shared<DIM>(g, q1, G);
  if (differ()) ++bad[7];
  const int kind[4] = {SURF_CHANDRASHEKAR, SURF_HLL, SURF_LLF, SURF_ROE};
  for (int i = 0; i < 4; ++i) {
    if (!try_surface_flux_shared<DIM, -1>(g, kind[i], q1, q2, n, G)) continue;
    FState<double, DIM> A, B;
    make_fstate<double, DIM>(g, q1, A);
    make_fstate<double, DIM>(g, q2, B);
    surface_flux_rt<double, DIM>(kind[i], g, A, B, n, F);
    if (differ()) ++bad[8 + i];
  }
}

__global__ void __launch_bounds__(kBlock) check_kernel(const GasT<double> g, unsigned long long *out) {
  unsigned long long bad[kChecks] = {};
  Rng r{(unsigned long long)blockIdx.x * kBlock + threadIdx.x + 1};
  r.s *= 0xD1342543DE82EF95ull;
  for (int it = 0; it < kPer; ++it) {
    const double x = r.scaled(400);
    if (!(ulps(rcp_refined(x), 1.0 / x) <= 1.0)) ++bad[0];
    const double num = r.scaled(200), den = r.scaled(200);
    if (!same(div_by(num, den, rcp_refined(den)), num / den)) ++bad[1];
    if (!same(div_by(-num, den, rcp_refined(den)), -num / den)) ++bad[1];
    const double x1 = r.scaled(100), y1 = r.partner(x1, 100), x2 = r.scaled(200), y2 = r.partner(x2, 200);
    const LogMeans m = log_means<LM_BRANCH>(x1, y1, x2, y2);
    const double a = log_mean(x1, y1), b = log_mean(x2, y2);
    if (!same(m.a, a) || !same(m.b, b) || !same(m.s2, x2 + y2)) ++bad[2];
    // for div_by: within 2^-44
    if (!(ulps(m.ia, 1.0 / a) <= 16.0) || !(ulps(m.ib, 1.0 / b) <= 16.0) || !(ulps(m.rs2, 1.0 / (x2 + y2)) <= 16.0))
      ++bad[3];
    const double yn = x1 * r.uniform(1.0 / 1.0195, 1.0195), zn = x2 * r.uniform(1.0 / 1.0195, 1.0195);
    const LogMeans s = log_means<LM_SERIES>(x1, yn, x2, zn);
    if (!same(s.a, log_mean(x1, yn)) || !same(s.b, log_mean(x2, zn))) ++bad[4];
    if (r.next() & 1) fluxes<2>(r, g, bad);
    else fluxes<3>(r, g, bad);
  }
  for (int i = 0; i < kChecks; ++i)
    if (bad[i]) atomicAdd(&out[i], bad[i]);
}

constexpr int kLogs = 1 << 20;
// arguments over 2^-400 .. 2^400, a quarter each around 1, around the branch
// of the logarithmic mean and within 1/4 .. 4
__global__ void log_kernel(double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kLogs) return;
  Rng r{(unsigned long long)i + 1};
  r.s *= 0xD1342543DE82EF95ull;
  double x = r.scaled(400);
  if (i % 4 == 1) x = 1.0 + ldexp(r.uniform(-1.0, 1.0), -1 - (int)(r.next() % 40));
  if (i % 4 == 2) x = r.uniform(1.02, 1.021);
  if (i % 4 == 3) x = exp2(r.uniform(-2.0, 2.0));
  if (i % 8 == 2) x = 1.0 / x;
  out[3 * i] = x;
  out[3 * i + 1] = log_normal(x);
  out[3 * i + 2] = log(x);
}

int main(int argc, char **argv) {
  if (argc != 2) return 2;
  GasT<double> g{};
  g.gamma = 1.4;
  g.gm1 = g.gamma - 1.0;
  g.gm1_inv = 1.0 / g.gm1;
  g.gm1_av_inv = 2.0 / (g.gamma + g.gamma - 2.0);
  g.inv_gm1 = 1.0 / (g.gamma - 1.0);
  unsigned long long *out, host[kChecks];
  if (cudaMalloc(&out, sizeof(host)) != cudaSuccess || cudaMemset(out, 0, sizeof(host)) != cudaSuccess) return 2;
  check_kernel<<<kGrid, kBlock>>>(g, out);
  if (cudaMemcpy(host, out, sizeof(host), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  int rc = 0;
  for (int i = 0; i < kChecks; ++i) {
    std::printf("%s %llu of %lld\n", kNames[i], host[i], (long long)kGrid * kBlock * kPer);
    if (host[i]) rc = 1;
  }
  double *logs;
  static double h[3 * kLogs];
  if (cudaMalloc(&logs, sizeof(h)) != cudaSuccess) return 2;
  log_kernel<<<kLogs / 256, 256>>>(logs);
  if (cudaMemcpy(h, logs, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  FILE *f = std::fopen(argv[1], "wb");
  if (!f || std::fwrite(h, 1, sizeof(h), f) != sizeof(h) || std::fclose(f)) return 2;
  return rc;
}
