// k_solve64.cu -- the implicit solve of CHF_FP64 on the tensor cores: the
// per-mode loop poiseuilleflow.f90:242-394 for every (kx, ky) but the (0,0)
// mode.
//
// The equations A x = B c + r (k_solve.cu's operators, the wall rows of B
// zero) are solved as a state plus an increment,
//   x = c + M c + X r,   X = A^-1,   M = X (B - A) = A^-1 B - I,
// as k_solve_mixed.cu does, in FP64 throughout: forming B c at the collocation
// points would cancel fourth derivatives of the coefficients against an O(c)
// result, M c has no such cancellation, and the step becomes two small
// matrix products per k^2 and parity.
//
// They are bound by the FP64 pipe (about 2 lane-operations per clock per SM)
// wherever it does them, so they run as exact digit products on mma.sync
// (digits64.cuh): set-up cuts M and X once per k^2 into eight planes of 8-bit
// digits against each row's largest entry, one byte per digit, so that an
// entry takes the 8 bytes it took in FP64; a step cuts the coefficients and
// the AB2 term of up to four modes of one k^2 (eight real columns, an n8
// operand) and multiplies.  The digits lose 2^-62 of the row's and of the
// column's largest value and the dropped levels about 2^-58 of their product.
// That is a loss only where the largest entry of a row takes no part: the
// columns of A^-1 that belong to the wall rows meet zeros (r vanishes there) but
// exceed v's other columns by 2^8 to 2^16 at large k^2, so they are left out of
// the digits.  With them A^-1 r came out 1e-14 to 1e-12 off (k^2 = 1e2 to 3e4,
// 128 intervals, dt 2e-4, re 180; relative to its largest value), without them
// 1e-17; plain FP64 gives 1e-16 (M c: 1e-17 against 1e-16).
//
// A CTA takes one run of at most 4 modes of one k^2 group (setup_inc_items).
// Warp (field, mode) reads the mode's coefficients and histories of one field
// once, finds the exponents of its four operands (even / odd coefficients,
// even / odd AB2 term) with warp reductions and writes their digits to shared
// memory in fragment order.  Then each warp takes strips of 16 rows of the
// four blocks (v even, v odd, omega even, omega odd) through M and X and adds
// the increment to the coefficients.  Wall-normal sizes are mostly 2^a + 1, so
// that the even blocks have 16 t + 1 rows: the last row and column stay out of
// the tiles (a fifth of them at 129 points) and are plain FP64.
//
// What it measures, 128 x 129 x 128 (box 4 pi x 2 x 4/3 pi, 3077 runs): 331 us
// (k_solve: 1314 with the recovery, which is 65 us here); DRAM 990 MB, 146 us
// at 6763 GB/s.  No unit is full (matrix pipe 33%, FP64 28%, issue 37%):
// 16 warps per SM wait on each other's latencies.  A strip's exponents, last
// columns and coefficients come before its products or stay in shared memory
// from the first part, because reading them after the products left three
// DRAM latencies per strip in the open (405 us); three CTAs per SM spill
// (474 us); operators brought to L2 during the first part change nothing
// (332 us); with a one-tile read of the operators the time is 310 us, without
// the products 288 us.
#include <algorithm>

#include "chf_internal.h"
#include "digits64.cuh"

namespace chf {

namespace {

constexpr int S64_MODES = 4;
constexpr int S64_THREADS = 256;      // warps: 4 modes x 2 fields
constexpr int S64_TILE = 520;         // words of a staged 16 x 8 tile: 8 planes x 32 lanes x 2, plus 8 to spread the banks
constexpr int S64_NAN = 100000;
constexpr int S64_BLOCK = 128;        // uint4 of a 16 x 16 operator tile: 4 per lane

struct Sol64Args {
  cd *v, *oy;
  const cd *rv, *u, *rg, *w;  // N^n and N^{n-1} at the Gauss-Lobatto points
  const uint4* mat;
  const short* exps;
  const double* ext;
  const int *group_start, *group_modes;
  const int2* items;
  Sol64Shape s;
  int N, NZ;
  long modes;
  double c3, c1;
};

__device__ __forceinline__ int biased_exp(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// ta 2^a + tb 2^b: aligned and added as integers (|ta|, |tb| < 2^60), one
// conversion, the exponent added to its bits
__device__ __forceinline__ double increment(long long ta, int a, long long tb, int b) {
  if (a >= S64_NAN / 2 || b >= S64_NAN / 2) return __longlong_as_double(0x7ff8000000000000ll);
  const int m = max(a, b);
  const long long t = (ta >> min(m - a, 63)) + (tb >> min(m - b, 63));
  const double v = (double)t;
  if (m < -960 || m > 900) return scalbn(v, m);
  return t == 0 ? 0.0 : __hiloint2double(__double2hiint(v) + (m << 20), __double2loint(v));
}

template <int ITER>  // k pairs per lane: 32 ITER >= 8 tiles
__global__ void __launch_bounds__(S64_THREADS, 2) k_solve64(const __grid_constant__ Sol64Args a) {
  // staged digit tiles [operand: coefficients, AB2 term][block][tile], then
  // the coefficients [block][mode][sh.pitch]
  extern __shared__ __align__(16) uint32_t dig[];
  __shared__ int s_exp[2][4][S64_MODES];    // e - 66 + shift of operand, block, mode (S64_NAN: not finite)
  __shared__ int s_shift[2][4][S64_MODES];
  __shared__ double2 s_last[2][4][S64_MODES];  // the operand's value at the block's last column
  __shared__ long s_mode[S64_MODES];
  const Sol64Shape& sh = a.s;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int2 it = a.items[blockIdx.x];
  const int grp = it.x, base = it.y, nm = min(S64_MODES, a.group_start[grp + 1] - base);
  const int N = a.N;
  const double* ext = a.ext + (size_t)grp * sh.ext_stride;
  double2* s_c = reinterpret_cast<double2*>(dig + (size_t)sh.staged_tiles * S64_TILE);
  const uint4* gmat = a.mat + (size_t)grp * sh.mat_stride;
  {
    // ---- the digits of one mode's field
    const int m = warp & 3, f = warp >> 2;
    const long mode = m < nm ? a.group_modes[base + m] : -1;
    if (lane == 0 && f == 0) s_mode[m] = mode;
    const cd* C = (f == 0 ? a.v : a.oy) + (mode < 0 ? 0 : mode);
    const cd* H = (f == 0 ? a.rv : a.rg) + (mode < 0 ? 0 : mode);   // N^n
    const cd* Ho = (f == 0 ? a.u : a.w) + (mode < 0 ? 0 : mode);    // N^{n-1}
    const int wall = f == 0 ? 2 : 1;
    auto coef = [&](int j) { return mode >= 0 && j <= N ? C[(size_t)j * a.modes] : cd{0.0, 0.0}; };
    auto term = [&](int p) {  // half of dt (3/2 N^n - 1/2 N^{n-1}) at point p
      const cd h = H[(size_t)p * a.modes], o = Ho[(size_t)p * a.modes];
      return cd{a.c3 * h.re - a.c1 * o.re, a.c3 * h.im - a.c1 * o.im};
    };
    auto fold = [&](int p, cd& e, cd& o) {  // even and odd part of the term at p and N - p
      e = o = cd{0.0, 0.0};
      if (mode < 0 || p < wall || p > N / 2) return;
      const cd x = term(p), y = term(N - p);
      e = cd{x.re + y.re, x.im + y.im};
      o = cd{x.re - y.re, x.im - y.im};
    };
    // x[set][i][comp of k, k + 1]: sets 0, 1 even / odd coefficients, 2, 3 even / odd term
    double x[4][ITER][4];
#pragma unroll
    for (int i = 0; i < ITER; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = 2 * (lane + 32 * i) + h;
        const cd ce = coef(2 * k), co = coef(2 * k + 1);
        cd re, ro;
        fold(k, re, ro);
        const cd y[4] = {ce, co, re, ro};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const bool in = k < sh.cols[t & 1];  // columns inside the tiles
          x[t][i][2 * h] = in ? y[t].re : 0.0;
          x[t][i][2 * h + 1] = in ? y[t].im : 0.0;
          if (t < 2 && in) s_c[((2 * f + t) * S64_MODES + m) * sh.pitch + k] = make_double2(y[t].re, y[t].im);
        }
      }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int par = t & 1, op = t >> 1, blk = 2 * f + par;
      int e = 1;
#pragma unroll
      for (int i = 0; i < ITER; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) e = max(e, biased_exp(x[t][i][c]));
      e = __reduce_max_sync(0xffffffffu, e);
      unsigned int sum = 0;
#pragma unroll
      for (int i = 0; i < ITER; ++i) {
        const int l = lane + 32 * i, tile = l >> 3;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const double u0 = x[t][i][c], u1 = x[t][i][2 + c];
          const long long x0 = fixed_of((uint32_t)__double2loint(u0), (uint32_t)__double2hiint(u0), e);
          const long long x1 = fixed_of((uint32_t)__double2loint(u1), (uint32_t)__double2hiint(u1), e);
          sum += ((unsigned int)(llabs(x0) >> 40) + 1u) + ((unsigned int)(llabs(x1) >> 40) + 1u);
          if (tile < sh.tiles[par]) {
            uint32_t w[8];
            digit_pairs(x0, x1, w);
            uint32_t* o = dig + (size_t)(sh.staged[op][blk] + tile) * S64_TILE + ((2 * m + c) * 4 + (l & 3)) * 2 + ((l >> 2) & 1);
#pragma unroll
            for (int p = 0; p < 8; ++p) o[p * 64] = w[p];
          }
        }
      }
      sum = __reduce_add_sync(0xffffffffu, sum);
      if (lane == 0) {
        // |level sum| < 2^(66 + b) for sum |value| < 2^(e + b) (re and im together)
        const int b = max(0, 32 - __clz(sum) - 21);
        s_shift[op][blk][m] = 7 + b;
        s_exp[op][blk][m] = e == 0x7ff ? S64_NAN : e - 1022 - 66 + 7 + b;
      }
    }
    // ---- the last row and column of a block of 16 t + 1
#pragma unroll
    for (int par = 0; par < 2; ++par) {
      if (!sh.ext[par] || mode < 0) continue;
      const int n = sh.n[par], blk = 2 * f + par, k = n - 1;
      const cd c = coef(2 * k + par);
      cd re, ro;
      fold(k, re, ro);
      const cd r = par ? ro : re;
      const double* rowm = ext + sh.ext_off[blk];  // [n] of M, [n] of X, then the columns
      const double* rowx = rowm + n;
      double sr = 0.0, si = 0.0;
#pragma unroll
      for (int i = 0; i < ITER; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int q = 2 * (lane + 32 * i) + h;
          if (q >= k) continue;
          const double mm = rowm[q], xx = rowx[q];
          sr = fma(mm, x[par][i][2 * h], fma(xx, x[2 + par][i][2 * h], sr));
          si = fma(mm, x[par][i][2 * h + 1], fma(xx, x[2 + par][i][2 * h + 1], si));
        }
      // the lower half-warp sums the real parts, the upper one the imaginary
      const bool up = lane >= 16;
      double sum = (up ? si : sr) + __shfl_xor_sync(0xffffffffu, up ? sr : si, 16);
      for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if ((lane & 15) == 0) {
        const double cc = up ? c.im : c.re;
        sum = fma(rowm[k], cc, fma(rowx[k], up ? r.im : r.re, sum));
        reinterpret_cast<double*>((f == 0 ? a.v : a.oy) + mode + (size_t)(2 * k + par) * a.modes)[up] = cc + sum;
      }
      if (lane == 0) {
        s_last[0][blk][m] = make_double2(c.re, c.im);
        s_last[1][blk][m] = make_double2(r.re, r.im);
      }
    }
  }
  __syncthreads();
  // ---- strips of 16 rows through M and X
  const int row = lane >> 2, q = lane & 3;  // the lane's rows row, row + 8 and its mode
  const long mode = s_mode[q];
  const short4* gexp = reinterpret_cast<const short4*>(a.exps) + (size_t)grp * sh.strips * 8 + row;
  for (int s = warp; s < sh.strips; s += S64_THREADS / 32) {
    __syncwarp();  // lanes without a mode left the last strip's stores early; mma takes whole warps
    int blk = 0;
    while (blk < 3 && s >= sh.strip0[blk + 1]) ++blk;
    const int i = s - sh.strip0[blk], par = blk & 1, T = sh.tiles[par], n = sh.n[par];
    const uint4* mp = gmat + lane + (size_t)(sh.mat0[blk] + 2 * T * i) * S64_BLOCK;
    long long prod[2][4];  // M c and X r of (row, re), (row, im), (row + 8, re), (row + 8, im)
    uint4 w[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) w[c] = __ldg(mp + c * 32);
    const short4 rexp = gexp[s * 8];  // of M and X in row, of M and X in row + 8
    double colm[2] = {0.0, 0.0}, colx[2] = {0.0, 0.0};  // the last column of M and X
    if (sh.ext[par]) {
      const double* col = ext + sh.ext_off[blk] + 2 * n + 16 * i + row;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        colm[h] = col[8 * h];
        colx[h] = col[n - 1 + 8 * h];
      }
    }
#pragma unroll 1
    for (int op = 0; op < 2; ++op) {
      float acc[8][4];
#pragma unroll
      for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[p][c] = 0.f;
#pragma unroll 1
      for (int t = 0; t < T; ++t) {
        const uint4 z[4] = {w[0], w[1], w[2], w[3]};
        mp += S64_BLOCK;
        if (t + 1 < T || op == 0) {  // the next tile, X's first one after M's last
#pragma unroll
          for (int c = 0; c < 4; ++c) w[c] = __ldg(mp + c * 32);
        }
        const uint2* b = reinterpret_cast<const uint2*>(dig + (size_t)(sh.staged[op][blk] + t) * S64_TILE) + lane;
        uint2 bf[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) bf[p] = b[p * 32];
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          const uint32_t w0 = (p & 1) ? z[p >> 1].z : z[p >> 1].x, w1 = (p & 1) ? z[p >> 1].w : z[p >> 1].y;
          const uint32_t af[4] = {to_half2(w0, 0x4140), to_half2(w1, 0x4140), to_half2(w0, 0x4342), to_half2(w1, 0x4342)};
#pragma unroll
          for (int r = 0; r + p < 8; ++r) mma16816(acc[p + r], af, bf[r].x, bf[r].y);
        }
      }
      const int sft = s_shift[op][blk][q];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float lev[8] = {acc[0][c], acc[1][c], acc[2][c], acc[3][c], acc[4][c], acc[5][c], acc[6][c], acc[7][c]};
        long long hi = 0, lo = 0;
        add_levels(lev, hi, lo);
        const long long t = (hi << (32 - sft)) + ((lo + (1ll << (sft - 1))) >> sft);
        if (op == 0) prod[0][c] = t;
        else prod[1][c] = t;
      }
    }
    if (mode < 0) continue;
    cd* dst = (blk < 2 ? a.v : a.oy) + mode;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = 16 * i + row + 8 * h;
      if (r >= sh.cols[par]) continue;  // tile rows past the block
      const int em = s_exp[0][blk][q] + (h ? rexp.z : rexp.x), ex = s_exp[1][blk][q] + (h ? rexp.w : rexp.y);
      double dr = increment(prod[0][2 * h], em, prod[1][2 * h], ex);
      double di = increment(prod[0][2 * h + 1], em, prod[1][2 * h + 1], ex);
      if (sh.ext[par]) {
        const double2 c = s_last[0][blk][q], t = s_last[1][blk][q];
        dr = fma(colm[h], c.x, fma(colx[h], t.x, dr));
        di = fma(colm[h], c.y, fma(colx[h], t.y, di));
      }
      const double2 c = s_c[(blk * S64_MODES + q) * sh.pitch + r];
      dst[(size_t)(2 * r + par) * a.modes] = cd{c.x + dr, c.y + di};
    }
  }
}

// ---------------------------------------------------------------------------
// Set-up, for groups g0 .. of a chunk: M in FP64, grid (groups, 4 blocks), as
// k_build_incr (k_solve_mixed.cu) forms it from the collocation matrices and
// X = A^-1; then the digits.
// ---------------------------------------------------------------------------
constexpr int BW64 = 32;  // columns of W = B - A staged per pass

__global__ void __launch_bounds__(256) k_build_m64(const double* __restrict__ t0, const double* __restrict__ t2,
                                                   const double* __restrict__ t4, const double* __restrict__ k2vals,
                                                   const double* __restrict__ xinv, SolveLayout sl, int N, double dt_re,
                                                   int g0, double* __restrict__ mout) {
  extern __shared__ __align__(16) double Wm[];  // W[q * BW64 + cc], column c0 + cc
  const int g = g0 + blockIdx.x, blk = blockIdx.y, NZ = N + 1;
  const bool isv = blk < 2, even = (blk % 2) == 0;
  const int n = even ? N / 2 + 1 : N / 2, r0 = isv ? 2 : 1;
  const BlockOffsets bo = block_offsets(sl);
  const size_t off = blk == 0 ? bo.ve : blk == 1 ? bo.vo : blk == 2 ? bo.we : bo.wo;
  const double* X = xinv + (size_t)g * sl.stride + off;  // column-major X[q * n + r]
  double* M = mout + (size_t)blockIdx.x * sl.stride + off;
  const double k2 = k2vals[g];
  for (int c0 = 0; c0 < n; c0 += BW64) {
    const int nc = min(BW64, n - c0);
    __syncthreads();
    for (int t = threadIdx.x; t < n * BW64; t += blockDim.x) {
      const int q = t / BW64, cc = t % BW64, j = even ? 2 * (c0 + cc) : 2 * (c0 + cc) + 1;
      double w = 0.0;
      if (q >= r0 && cc < nc) {
        const size_t p = (size_t)q + (size_t)NZ * j;
        w = isv ? dt_re * (t4[p] - 2.0 * k2 * t2[p] + k2 * k2 * t0[p]) : dt_re * (t2[p] - k2 * t0[p]);
      } else if (cc < nc) {
        w = (isv && q == 1) ? -(double)j * (double)j : -1.0;
      }
      Wm[t] = w;
    }
    __syncthreads();
    // four columns per thread: one read of X serves them
    const int quads = (nc + 3) / 4;
    for (int t = threadIdx.x; t < n * quads; t += blockDim.x) {
      const int c = 4 * (t / n), r = t % n;
      double acc[4] = {0.0, 0.0, 0.0, 0.0};
      for (int q = 0; q < n; ++q) {
        const double x = X[(size_t)q * n + r];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = fma(x, Wm[q * BW64 + c + i], acc[i]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (c + i < nc) M[(size_t)(c0 + c + i) * n + r] = acc[i];
    }
  }
}

// Digits of the strips: grid (groups, strips), 256 threads.  Each operand's
// 16 rows: their exponents, then per tile and lane 4 uint4 with the digit
// bytes of rows lane / 4, + 8 at k = 2 (lane % 4), + 1, + 8, + 9; plus the
// block's last row and column in FP64 where they stay out of the tiles.
__global__ void __launch_bounds__(256) k_digits_solve64(const double* __restrict__ minc, const double* __restrict__ xinv,
                                                        SolveLayout sl, Sol64Shape sh, int g0, uint4* __restrict__ mat,
                                                        short* __restrict__ exps, double* __restrict__ ext) {
  __shared__ int s_e[2][16];
  const int gl = blockIdx.x, g = g0 + gl, s = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int blk = 0;
  while (blk < 3 && s >= sh.strip0[blk + 1]) ++blk;
  const int i = s - sh.strip0[blk], par = blk & 1, T = sh.tiles[par], n = sh.n[par], cols = sh.cols[par];
  const BlockOffsets bo = block_offsets(sl);
  const size_t off = blk == 0 ? bo.ve : blk == 1 ? bo.vo : blk == 2 ? bo.we : bo.wo;
  const double* src[2] = {minc + (size_t)gl * sl.stride + off, xinv + (size_t)g * sl.stride + off};
  const int first[2] = {0, blk < 2 ? 2 : 1};  // A^-1's columns of the wall rows, whose r is zero, stay out
  if (tid < 32) s_e[tid >> 4][tid & 15] = 1;
  __syncthreads();
  for (int op = 0; op < 2; ++op) {
    const int r = 16 * i + (tid & 15);
    int e = 0;
    if (r < cols)
      for (int c = first[op] + (tid >> 4); c < cols; c += 16) e = max(e, biased_exp(src[op][(size_t)c * n + r]));
    atomicMax(&s_e[op][tid & 15], e);
  }
  __syncthreads();
  // a row's power of two
  if (tid < 32)
    exps[(((size_t)g * sh.strips + s) * 8 + (tid & 7)) * 4 + 2 * ((tid >> 3) & 1) + (tid >> 4)] =
        (short)(s_e[tid >> 4][tid & 15] - 1022);
  uint4* out = mat + (size_t)g * sh.mat_stride + (size_t)(sh.mat0[blk] + 2 * T * i) * S64_BLOCK + lane;
  for (int t = warp; t < 2 * T; t += 8) {
    const int op = t / T, kt = t - op * T;
    uint32_t w[2][8];
    for (int h = 0; h < 2; ++h) {
      const int r = 16 * i + lane / 4 + 8 * h;
      long long x[4];
      for (int c = 0; c < 4; ++c) {
        const int k = 16 * kt + 2 * (lane & 3) + (c & 1) + 8 * (c >> 1);
        const double v = r < cols && k >= first[op] && k < cols ? src[op][(size_t)k * n + r] : 0.0;
        x[c] = fixed_of((uint32_t)__double2loint(v), (uint32_t)__double2hiint(v), s_e[op][lane / 4 + 8 * h]);
      }
      digit_bytes(x, w[h]);
    }
    for (int c = 0; c < 4; ++c)
      out[(size_t)t * S64_BLOCK + c * 32] = make_uint4(w[0][2 * c], w[1][2 * c], w[0][2 * c + 1], w[1][2 * c + 1]);
  }
  if (i == 0 && sh.ext[par]) {
    double* o = ext + (size_t)g * sh.ext_stride + sh.ext_off[blk];
    for (int k = tid; k < n; k += 256) {
      for (int op = 0; op < 2; ++op) {
        o[op * n + k] = src[op][(size_t)k * n + n - 1];                               // the last row
        if (k < n - 1) o[2 * n + op * (n - 1) + k] = src[op][(size_t)(n - 1) * n + k];  // the last column
      }
    }
  }
}

}  // namespace

Sol64Shape solve64_shape(int N) {
  Sol64Shape s{};
  int staged = 0, strip = 0, mat = 0, ext = 0;
  for (int par = 0; par < 2; ++par) {
    const int n = par ? N / 2 : N / 2 + 1;
    s.n[par] = n;
    s.ext[par] = n > 16 && n % 16 == 1;
    s.cols[par] = s.ext[par] ? n - 1 : n;
    s.tiles[par] = (s.cols[par] + 15) / 16;
  }
  for (int blk = 0; blk < 4; ++blk) {
    const int par = blk & 1, T = s.tiles[par];
    for (int op = 0; op < 2; ++op) {
      s.staged[op][blk] = staged;
      staged += T;
    }
    s.strip0[blk] = strip;
    strip += T;
    s.mat0[blk] = mat;
    mat += 2 * T * T;
    s.ext_off[blk] = ext;
    if (s.ext[par]) ext += 4 * s.n[par];
  }
  s.strips = strip;
  // rows 1 and 2 apart and modes apart by 2 (mod 8) of the 16-byte banks
  s.pitch = (s.n[0] + 5) / 8 * 8 + 2;
  s.staged_tiles = staged;
  s.mat_stride = (size_t)mat * S64_BLOCK;
  s.ext_stride = std::max(1, ext);
  return s;
}

// CHF_FP64 takes this path where k_solve's CTAs (runs of 2 modes and the (0,0)
// mode) would be more than one per SM: below that both are bound by latency,
// and k_solve is one kernel instead of three and needs no further set-up.
// Whole steps, this path against k_solve, on the same transforms: 32 x 17 x 32
// 85 / 88 us, 32^3 112 / 118 (216 / 241 with three such channels at a time),
// 64 x 65 x 64 462 / 544, 128 x 129 x 128 2717 / 3600; with fewer CTAs than
// SMs 16 x 65 x 16 131 / 125, 16 x 65 x 4 121 / 115, 24 x 21 x 12 78 / 80.
// CHF_MIXED_F64SOLVE stays with k_solve: its FP32 front turns any change of
// the state's last bit into another rounding of the next step.
//
// The digits of M and X take twice the bytes of the inverses (128 x 129 x 128:
// 0.85 against 0.42 GB), which go once they are cut, all but the (0,0) mode's.
// Where the device cannot hold them (spare_memory), k_solve serves as well.
bool solve64(const Handle* h) { return h->s64_mat != nullptr; }

int setup_solve64(Handle* h) {
  if (h->cfg.precision != CHF_FP64 || h->n_inc_items[0] + 1 <= h->num_sms) return CHF_OK;
  const Sol64Shape s = solve64_shape(h->d.N);
  const size_t all = (size_t)h->nk2, group = sizeof(double) * h->sl.stride;
  const int chunk = std::min(h->nk2, 1024);  // groups whose M is held in FP64 at a time
  const size_t size[4] = {sizeof(uint4) * s.mat_stride * all, sizeof(short) * 32 * s.strips * all,
                          sizeof(double) * s.ext_stride * all, group * chunk};
  if (!spare_memory(h, size[0] + size[1] + size[2] + size[3])) return CHF_OK;
  void* mem[4] = {};
  auto drop = [&] {
    for (void* p : mem) cudaFree(p);
    cudaGetLastError();
  };
  for (int i = 0; i < 4; ++i)
    if (cudaMalloc(&mem[i], size[i]) != cudaSuccess) {
      drop();
      return CHF_OK;
    }
  uint4* const mat = static_cast<uint4*>(mem[0]);
  short* const exps = static_cast<short*>(mem[1]);
  double *const ext = static_cast<double*>(mem[2]), *const minc = static_cast<double*>(mem[3]);
  const size_t smem = sizeof(double) * (size_t)s.n[0] * BW64;
  for (int g0 = 0; g0 < h->nk2; g0 += chunk) {
    const int ng = std::min(chunk, h->nk2 - g0);
    k_build_m64<<<dim3(ng, 4), 256, smem, h->stream>>>(h->t0, h->t2, h->t4, h->k2vals, h->xinv, h->sl, h->d.N,
                                                       h->cfg.dt / h->cfg.re, g0, minc);
    k_digits_solve64<<<dim3(ng, s.strips), 256, 0, h->stream>>>(minc, h->xinv, h->sl, s, g0, mat, exps, ext);
  }
  // the (0,0) mode's inverse alone, in place of all
  double* keep = nullptr;
  if (cudaMalloc((void**)&keep, group) != cudaSuccess) {
    drop();
    return CHF_OK;
  }
  if (!cuda_ok(h, cudaGetLastError(), "solve set-up") ||
      !cuda_ok(h, cudaMemcpyAsync(keep, h->xinv + h->sl.stride * all, group, cudaMemcpyDeviceToDevice, h->stream),
               "solve set-up") ||
      !cuda_ok(h, cudaStreamSynchronize(h->stream), "solve set-up")) {
    drop();
    cudaFree(keep);
    return CHF_E_CUDA;
  }
  cudaFree(minc);
  cudaFree(h->xinv);
  h->xinv = keep;
  h->xinv_first = h->nk2;
  h->s64 = s;
  h->s64_mat = mat;
  h->s64_exp = exps;
  h->s64_ext = ext;
  return CHF_OK;
}

int launch_solve64(Handle* h) {
  const Sol64Shape& s = h->s64;
  Sol64Args a{};
  a.v = h->f[F_V];
  a.oy = h->f[F_OY];
  a.rv = h->f[F_RV];
  a.u = h->f[F_U];
  a.rg = h->f[F_RG];
  a.w = h->f[F_W];
  a.mat = h->s64_mat;
  a.exps = h->s64_exp;
  a.ext = h->s64_ext;
  a.group_start = h->group_start;
  a.group_modes = h->group_modes;
  a.items = h->inc_items;
  a.s = s;
  a.N = h->d.N;
  a.NZ = h->d.NZ;
  a.modes = h->d.modes();
  a.c3 = 0.75 * h->cfg.dt;
  a.c1 = 0.25 * h->cfg.dt;
  const size_t smem = sizeof(uint32_t) * S64_TILE * (size_t)s.staged_tiles + sizeof(double2) * 4 * S64_MODES * s.pitch;
  auto kern = std::max(s.tiles[0], s.tiles[1]) <= 4 ? k_solve64<1> : k_solve64<2>;
  if (!cuda_ok(h, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "k_solve64 smem"))
    return CHF_E_CUDA;
  cudaEvent_t ev;
  prof_begin(h, K_SOLVE, &ev);
  kern<<<h->n_inc_items[1], S64_THREADS, smem, h->stream>>>(a);
  prof_end(h, K_SOLVE, ev);
  return cuda_ok(h, cudaGetLastError(), "k_solve64") ? CHF_OK : CHF_E_CUDA;
}

}  // namespace chf
