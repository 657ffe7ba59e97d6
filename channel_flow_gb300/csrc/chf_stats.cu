// chf_stats.cu -- flow statistics on the GPU (statistics, poiseuilleflow.f90:2666-3198).
//
// The reference transforms u, v, w to the physical nnx x nny x (nz+1) grid
// (transform(1), unpadded) at every outputstep and forms, per Gauss-Lobatto
// plane z_k, the plane means <u>, <v>, <w> and the covariances
// <u'u'>, <v'v'>, <w'w'>, <u'v'>, <u'w'>, <v'w'> (:2945-3060), the physical
// kinetic energy sum (:2786-2800) and from these the wall shear velocities,
// Re_tau, Re_c and Re_b (:3150-3190).  Plane averages of products of
// band-limited fields are exact spectral sums (Parseval; the products
// cannot alias onto the zero mode because the spanwise Nyquist slot is
// empty), so here they are computed without any in-plane transform:
//   <f'g'>(z_k) = sum over modes (kx, ky) != (0, 0) of w_kx Re(f^(z_k) conj(g^(z_k))),
// with w_kx = 1 for kx = 0 and 2 for kx > 0 (the half spectrum in x), and
// <f>(z_k) = Re f^_{00}(z_k).  The only transform is Chebyshev coefficients
// -> Gauss-Lobatto values, as exact digit products (k_dft64.cu).  A whole call
// at 128^3 takes 182 us, with the FFTs of these lines and weights in the sums it
// took 466; at 32^3 48 / 58 us.
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "chf_internal.h"

using namespace chf;

struct chf_handle : public Handle {};

namespace {

constexpr int ST_THREADS = 256;
constexpr int NSTAT = 10;      // per plane: <u>,<v>,<w>, uu,vv,ww, uv,uw,vw, energy density

// one CTA per plane k: means, covariances and sum_modes w (|u|^2+|v|^2+|w|^2)
__global__ void __launch_bounds__(ST_THREADS) k_stat_sum(const cd* __restrict__ gl, Dims d, double* __restrict__ out) {
  const int k = blockIdx.x, NZ = d.NZ;
  const long modes = d.modes();
  const cd* U = gl + ((size_t)0 * NZ + k) * modes;
  const cd* V = gl + ((size_t)1 * NZ + k) * modes;
  const cd* W = gl + ((size_t)2 * NZ + k) * modes;
  // uu vv ww uv uw vw, the modes of kx = 0 (weight 1) before those of kx > 0
  // (weight 2): 12 FP64 operations per mode and no weight to multiply
  double acc[6] = {0, 0, 0, 0, 0, 0};
  auto add = [&](long m) {
    const cd a = U[m], b = V[m], c = W[m];
    acc[0] = fma(a.re, a.re, fma(a.im, a.im, acc[0]));
    acc[1] = fma(b.re, b.re, fma(b.im, b.im, acc[1]));
    acc[2] = fma(c.re, c.re, fma(c.im, c.im, acc[2]));
    acc[3] = fma(a.re, b.re, fma(a.im, b.im, acc[3]));
    acc[4] = fma(a.re, c.re, fma(a.im, c.im, acc[4]));
    acc[5] = fma(b.re, c.re, fma(b.im, c.im, acc[5]));
  };
  const long nyq0 = (long)d.NYQ * d.KX, nyq1 = nyq0 + d.KX;  // the spanwise Nyquist slot is left out
  double zero[6];
  for (int ky = threadIdx.x; ky < d.KY; ky += blockDim.x)
    if (ky != d.NYQ && ky > 0) add((long)ky * d.KX);  // (0, 0) is not a fluctuation
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    zero[q] = acc[q];
    acc[q] = 0.0;
  }
  for (long m = threadIdx.x; m < modes; m += blockDim.x)
    if ((unsigned int)m % (unsigned int)d.KX != 0 && (m < nyq0 || m >= nyq1)) add(m);
#pragma unroll
  for (int q = 0; q < 6; ++q) acc[q] = fma(2.0, acc[q], zero[q]);
  __shared__ double red[ST_THREADS / 32][6];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    double x = acc[q];
    for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
    if (lane == 0) red[warp][q] = x;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double x = 0.0;
    for (int q = 0; q < ST_THREADS / 32; ++q) x += red[q][threadIdx.x];
    out[(size_t)k * NSTAT + 3 + threadIdx.x] = x;
    red[0][threadIdx.x] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const cd a = U[0], b = V[0], c = W[0];
    out[(size_t)k * NSTAT + 0] = a.re;
    out[(size_t)k * NSTAT + 1] = b.re;
    out[(size_t)k * NSTAT + 2] = c.re;
    const double mean = (a.re * a.re + a.im * a.im) + (b.re * b.re + b.im * b.im) + (c.re * c.re + c.im * c.im);
    out[(size_t)k * NSTAT + 9] = mean + red[0][0] + red[0][1] + red[0][2];
  }
}

}  // namespace

extern "C" int chf_statistics(chf_handle* h, double* profiles, chf_stats* out) {
  if (!h || !out) return CHF_E_INVALID;
  if (!h->uploaded) {
    h->err = "chf_statistics before chf_upload_state";
    return CHF_E_STATE;
  }
  if (!cuda_ok(h, cudaSetDevice(h->device), "cudaSetDevice")) return CHF_E_CUDA;
  const Dims& d = h->d;
  const int N = d.N, NZ = d.NZ;
  const size_t gl_elems = (size_t)3 * NZ * d.modes();
  if (!h->stats_buf) {  // first call: GL values of three fields + plane sums
    const size_t bytes = sizeof(cd) * gl_elems + sizeof(double) * (size_t)NZ * NSTAT;
    if (!cuda_ok(h, cudaMalloc(&h->stats_buf, bytes), "statistics buffer")) return CHF_E_NOMEM;
  }
  cd* gl = static_cast<cd*>(h->stats_buf);
  double* sums = reinterpret_cast<double*>(gl + gl_elems);
  const cd* in[3] = {h->f[F_U], h->f[F_V], h->f[F_W]};
  cd* val[3] = {gl, gl + gl_elems / 3, gl + 2 * (gl_elems / 3)};
  int rc;
  if ((rc = setup_tf_out(h)) != CHF_OK || (rc = launch_tf_gl(h, in, val, 3)) != CHF_OK) return rc;
  k_stat_sum<<<NZ, ST_THREADS, 0, h->stream>>>(gl, d, sums);
  if (!cuda_ok(h, cudaGetLastError(), "statistics kernels")) return CHF_E_CUDA;
  std::vector<double> S((size_t)NZ * NSTAT), au0(2 * (size_t)NZ);
  if (!cuda_ok(h, cudaMemcpyAsync(S.data(), sums, sizeof(double) * S.size(), cudaMemcpyDeviceToHost, h->stream),
               "statistics download") ||
      !cuda_ok(h, cudaMemcpyAsync(au0.data(), h->mean[M_AU0], sizeof(double) * au0.size(),
                                  cudaMemcpyDeviceToHost, h->stream),
               "statistics download") ||
      !cuda_ok(h, cudaStreamSynchronize(h->stream), "statistics sync"))
    return CHF_E_CUDA;
  const double re = h->cfg.re, pi = 3.14159265358979323846;
  std::vector<double> z(NZ);
  for (int k = 0; k < NZ; ++k) z[k] = std::cos(pi * k / N);
  // wall stress: d<u>/dz / re at z = +1 (k = 0) and z = -1 (k = nz), where the
  // Reynolds stress vanishes; T_n'(1) = n^2, T_n'(-1) = (-1)^(n+1) n^2
  double dtop = 0.0, dbot = 0.0, ub = 0.0;
  for (int n = 0; n < NZ; ++n) {
    const double a = au0[2 * n], n2 = (double)n * n;
    dtop += a * n2;
    dbot += ((n % 2) ? a : -a) * n2;
    if (n % 2 == 0) ub += a / (1.0 - n2);
  }
  out->u_tau_top = std::sqrt(std::fabs(dtop / re));
  out->u_tau_bottom = std::sqrt(std::fabs(dbot / re));
  out->re_tau_top = out->u_tau_top * re;
  out->re_tau_bottom = out->u_tau_bottom * re;
  out->re_centre = S[(size_t)(N / 2) * NSTAT + 0] * re;
  double ubr = 0.0;  // the reference's half-channel rectangle rule (:3176-3179)
  for (int k = N / 2; k <= N - 1; ++k) ubr += S[(size_t)k * NSTAT + 0] * std::fabs(z[k + 1] - z[k]);
  out->re_bulk = 2.0 * ubr * re;
  out->bulk_velocity = ub;
  double e = 0.0;
  for (int k = 0; k < NZ; ++k) e += S[(size_t)k * NSTAT + 9];
  out->energy = 0.5 * (double)d.nnx * (double)d.nny * e;
  if (profiles)
    for (int k = 0; k < NZ; ++k) {
      profiles[0 * NZ + k] = z[k];
      for (int q = 0; q < 9; ++q) profiles[(size_t)(q + 1) * NZ + k] = S[(size_t)k * NSTAT + q];
    }
  return CHF_OK;
}
