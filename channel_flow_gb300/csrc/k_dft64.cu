// k_dft64.cu -- the transforms of getnonlinear (poiseuilleflow.f90:1380-1612)
// in FP64 on the tensor cores.
//
// Why: GB300 retires about 2 FP64 lane-operations per clock per SM, and the
// FP64 FFTs of k_nonlinear.cu are bound by them.  mma.sync on 16-bit operands
// sustains 595 TFLOP/s (measured), so a dense transform of a short line as
// products of exact digits is several times faster than its FFT: 36 digit
// products make one FP64 product, 8.3e12 of which per second stand against
// 0.63e12 FP64 operations.
//
// What: every transform of the path is a real matrix on real lines, and the
// mirror symmetry of its points halves it twice,
//   E_n = sum_k C[n][k] u_k,   O_n = sum_k S[n][k] v_k,
// where (u, v) are the even / odd coefficients of a Chebyshev series, the
// sum / difference of mirrored points or modes, or the real / imaginary
// parts, and the outputs n and -n are E + O and E - O (k_tf's modes).
//
// How: a line is scaled by the power of two above its largest |value| into
// 62-bit integers, folded as integers (exact) and written as eight digits of
// 8 bits, x = sum_p d_p 256^(7-p) with d_p in [-128, 127]; the matrix likewise.
// Digits are exact in FP16, products of level p + q = 0..7 accumulate in FP32
// as integers below 2^24 (at most 8 products of 2^14 over 128 k; longer lines
// are summed in segments), so a level sum is exact, and the levels are
// combined in 64-bit integers and converted once.  What is lost is the
// rounding of the inputs at 2^-62 and the dropped levels, about 2^-58 of the
// line's largest value, and the final rounding at 2^-57 of the sum of its
// magnitudes: below the rounding of an FP64 FFT of the same line (2^-53 per
// stage of its norm).
//
// A CTA takes 16 real lines: its threads load each value once, keep the raw
// bits in shared memory that the digits will fill, find the lines' exponents
// and replace the bits by FP16 digits in the layout that ldmatrix reads as the
// A operand of m16n8k16; four warps then multiply the lines by 8 outputs at a
// time, the matrix digits coming from global memory (L2) in fragment order.
// The product of a tile waits on shared-memory and L2 reads as much as on the
// tensor pipe: 57% active in TF_XINV at 128^3, 66% of L1's data bandwidth.
// Measured and not taken: tiles of 16 outputs per warp (half the reads, fewer
// warps: 20% slower), digits kept as bytes and converted on each read (5%
// slower), the matrix digits of the next step loaded ahead (equal), 5 or 6
// CTAs per SM at fewer registers (equal), the last tiles' steps dealt to all four
// warps (4% slower), the Lamb products in TF_XFWD's loads (437 -> 634 us for the
// two), integer instead of FP64-pipe conversions of the outputs (5% slower).
// Parts switched off in TF_XINV, of 632 us: loads 46, digits 50, stores 110
// (conversions 40), products 280.
// At 128 x 129 x 128 (product grid 200), against the FFT kernels: z inverse
// 1.52 -> 0.30 ms, y inverse 0.68 -> 0.40, x with products 1.92 -> 1.04, y
// forward 0.36 -> 0.25, z forward with curl and Gauss-Lobatto values 1.17 ->
// 0.32; the errors against 64 bits of every array are equal or smaller (grids
// of 4 to 192 points a side).
#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>

#include "chf_internal.h"
#include "digits64.cuh"

namespace chf {

namespace {

constexpr int TF_THREADS = 128;
constexpr int TF_CTAS = 4;
constexpr int TF_LINES = 16;  // real lines per CTA (y: 8 complex ones)
constexpr int TF_SEG = 8;     // k16 steps whose level sums stay below 2^24

// modes of k_tf: input (u, v) of index k, and where outputs go
enum TfMode {
  TF_Z,     // coefficients 2k, 2k + 1 -> values at points n and M - n: E + O, E - O
  TF_YINV,  // modes k + -k, k - -k of a complex line -> points n, L - n: E + i O, E - i O
  TF_XINV,  // Re, Im of mode k -> real points n, L - n: E - O, E + O
  TF_XFWD,  // points k, L - k of a real line -> modes n: E - i O
  TF_YFWD,  // points k, L - k of a complex line -> modes n, -n: E - i O, E + i O
  TF_Z2     // values at points k, M - k -> coefficients 2n: E, 2n + 1: O
};

struct TfArgs {
  const double* in[6];
  double* out[6];
  const uint4* mat;  // digit fragments: E tiles, then O tiles (k_tf_matrix)
  TfShape s;
  long lines;        // real lines (y: complex)
  int nfields;
  double scale;  // of the outputs (TF_YFWD, TF_Z2; 1 otherwise)
  Dims d;
};

// the digits of eight integers as FP16: word[p][j] holds digit p of x[2j], x[2j + 1]
__device__ __forceinline__ void digit_halves(const long long* x, uint32_t (&word)[8][4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t w[8];
    digit_pairs(x[2 * j], x[2 * j + 1], w);
#pragma unroll
    for (int p = 0; p < 8; ++p) word[p][j] = w[p];
  }
}

// t 2^n, the exponent added to the conversion's (n in the range where every
// result is normal; `scale` serves the other lines: the largest times 1, the
// smallest, whose factor is no double, in two steps)
constexpr int TF_LARGE = INT_MIN, TF_SMALL = INT_MIN + 1;
__device__ __forceinline__ double scaled(long long t, int n, double scale) {
  const double v = (double)t;
  if (n <= TF_SMALL) return n == TF_LARGE ? v * scale : t == 0 ? 0.0 : v * scale * 0x1p-200;
  return t == 0 ? 0.0 : __hiloint2double(__double2hiint(v) + (n << 20), __double2loint(v));
}

template <int MODE>
__global__ void __launch_bounds__(TF_THREADS, TF_CTAS) k_tf(const __grid_constant__ TfArgs a) {
  constexpr bool YM = MODE == TF_YINV || MODE == TF_YFWD;
  constexpr bool FOLD = YM || MODE == TF_XFWD || MODE == TF_Z2;
  // digit blocks [8 planes][KS] of 512 bytes: 16 lines x 16 k as the four 8 x 8
  // matrices of ldmatrix, (k half, line half) major, rows of 16 bytes
  extern __shared__ __align__(16) uint4 dig[];
  __shared__ int s_emax[TF_LINES];
  __shared__ unsigned int s_sum[TF_LINES];
  __shared__ double s_scale[TF_LINES];
  __shared__ int s_shift[TF_LINES], s_exp[TF_LINES];
  const Dims& d = a.d;
  const TfShape& sh = a.s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = (int)(blockIdx.x % a.nfields);
  const long l0 = (long)(blockIdx.x / a.nfields) * (YM ? TF_LINES / 2 : TF_LINES);
  const int KS = sh.ks_e + sh.ks_o;
  // the thread's line: y lines lie re, im in memory, and go to rows j, j + 8
  const int ll = tid & 15;
  const int slot = YM ? ((ll & 1) << 3) + (ll >> 1) : ll;
  const int el = YM ? ll >> 1 : ll;  // its exponent entry (re and im share one)
  const long line = l0 + (YM ? ll >> 1 : ll);
  const bool live = line < a.lines;
  const double* src = a.in[f];
  size_t stride = 0;
  if constexpr (MODE == TF_Z || MODE == TF_Z2) {
    src += live ? line : 0;
    stride = 2 * (size_t)d.modes();
  } else if constexpr (YM) {
    const long p = live ? line / d.KX : 0;
    const int kx = live ? (int)(line - p * d.KX) : 0;
    src += 2 * ((size_t)p * (MODE == TF_YINV ? d.KY : d.PY) * d.KX + kx) + (ll & 1);
    stride = 2 * (size_t)d.KX;
  } else {
    src += (size_t)(live ? line : 0) * (MODE == TF_XINV ? 2 * d.KX : d.PX);
    stride = 1;
  }
  // u, v of index k
  auto fetch = [&](int k, double& u, double& v) {
    u = v = 0.0;
    if (!live || k >= sh.k_e) return;
    if constexpr (MODE == TF_Z) {
      u = src[(size_t)(2 * k) * stride];
      if (k < sh.k_o) v = src[(size_t)(2 * k + 1) * stride];
    } else if constexpr (MODE == TF_XINV) {
      const double2 z = *reinterpret_cast<const double2*>(src + 2 * k);
      u = z.x;
      v = k == 0 ? 0.0 : z.y;  // imaginary part of the streamwise mean dropped
    } else {
      // the mirror of k; none for the fixed points of the reflection
      const int m = MODE == TF_YINV ? (k == 0 ? 0 : d.KY - k) : MODE == TF_Z2 ? d.MZ - k : (k == 0 ? 0 : sh.L - k);
      u = src[(size_t)k * stride];
      if (m > k) v = src[(size_t)m * stride];
    }
  };
  // u, v of k0 .. k0 + 7 of a real line (TF_XFWD), two points per load (nine
  // loads for sixteen: 350 -> 322 us at 128 x 129 x 128).  L is even, so the
  // mirrors of an odd k and the even one above it make an aligned pair.
  auto fetch_pairs = [&](int k0, double (&u)[8], double (&v)[8]) {
    const int last = live ? sh.k_e - 1 : -1, m0 = sh.L - k0;  // last = L / 2, its own mirror
    const double2* pairs = reinterpret_cast<const double2*>(src);
    double2 a[4], b[5];  // points k0 + 2 i, + 1; points m0 - 2 i, + 1
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = k0 + 2 * i <= last ? pairs[(k0 >> 1) + i] : make_double2(0.0, 0.0);
#pragma unroll
    for (int i = 0; i < 5; ++i)
      b[i] = k0 + 2 * i > 0 && k0 + 2 * i - 1 <= last ? pairs[(m0 >> 1) - i] : make_double2(0.0, 0.0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = k0 + i;
      u[i] = k <= last ? ((i & 1) ? a[i >> 1].y : a[i >> 1].x) : 0.0;
      v[i] = k > 0 && k < last ? ((i & 1) ? b[(i + 1) >> 1].y : b[i >> 1].x) : 0.0;
    }
  };
  // 16-byte piece of (plane, octet of k) of the thread's line; O octets follow E's
  auto piece = [&](int plane, int octet) {
    return (plane * KS + (octet >> 1)) * 32 + (octet & 1) * 16 + slot;
  };
  if (tid < TF_LINES) {
    s_emax[tid] = 1;
    s_sum[tid] = 0u;
  }
  // ---- the values' bits into pieces of planes 0..3, the largest exponent
  const int oct_e = 2 * sh.ks_e, oct_o = 2 * sh.ks_o, octs = max(oct_e, oct_o);
  int emax = 0;
  for (int o = tid >> 4; o < octs; o += TF_THREADS / 16) {
    double u[8], v[8];
    if constexpr (MODE == TF_XFWD) {
      fetch_pairs(8 * o, u, v);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) fetch(8 * o + i, u[i], v[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      emax = max(emax, max((__double2hiint(u[i]) >> 20) & 0x7ff, (__double2hiint(v[i]) >> 20) & 0x7ff));
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      if (o < oct_e) *reinterpret_cast<double2*>(&dig[piece(p, o)]) = make_double2(u[2 * p], u[2 * p + 1]);
      if (o < oct_o) *reinterpret_cast<double2*>(&dig[piece(p, oct_e + o)]) = make_double2(v[2 * p], v[2 * p + 1]);
    }
  }
  __syncthreads();
  atomicMax(&s_emax[el], emax);
  __syncthreads();
  emax = s_emax[el];
  // ---- digits, and the sum of |value| (in 2^-21 of 2^e, rounded up)
  unsigned int sum = 0;
  for (int o = tid >> 4; o < octs; o += TF_THREADS / 16) {
    long long U[8], V[8];
    auto integers = [&](long long* X, int octet) {
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const uint4 w = dig[piece(p, octet)];
        X[2 * p] = fixed_of(w.x, w.y, emax);
        X[2 * p + 1] = fixed_of(w.z, w.w, emax);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) sum += (unsigned int)(llabs(X[i]) >> 40) + 1u;
    };
    auto digits = [&](const long long* X, int octet) {
      uint32_t w[8][4];
      digit_halves(X, w);
#pragma unroll
      for (int p = 0; p < 8; ++p) dig[piece(p, octet)] = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
    };
#pragma unroll
    for (int i = 0; i < 8; ++i) U[i] = V[i] = 0;
    if (o < oct_e) integers(U, o);
    if (o < oct_o) integers(V, oct_e + o);
    if (FOLD) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const long long t = U[i] - V[i];
        U[i] += V[i];
        V[i] = t;
      }
    }
    if (o < oct_e) digits(U, o);
    if (o < oct_o) digits(V, oct_e + o);
  }
  atomicAdd(&s_sum[el], sum);
  __syncthreads();
  // ---- per line: |level sum| < 2^(67 + b) for sum |value| < 2^(e + b).  The
  // shift 10 + b leaves 57 bits of that, and on a constant line of K values
  // (2^b >= K / 2) it exceeds twice the most that the dropped levels can hold,
  // 7 K 2^14 / 256 units: sums that are zero come out as zero.  Then the
  // outputs' scale (NaN for non-finite lines).
  if (tid < TF_LINES) {
    const int e = s_emax[tid];
    const int b = max(0, 32 - __clz(s_sum[tid]) - 21), n = e - 1022 + sh.f - 57 + b;
    s_shift[tid] = 10 + b;
    s_exp[tid] = n >= 900 ? TF_LARGE : n <= -960 ? TF_SMALL : n;
    s_scale[tid] = e == 0x7ff ? __longlong_as_double(0x7ff8000000000000ll) : scalbn(1.0, n <= -960 ? n + 200 : n);
  }
  __syncthreads();
  // ---- products: warp = every fourth tile of 8 outputs
  const int row = lane >> 2, cq = lane & 3;
  const int ea = row, eb = YM ? ea : ea + 8;
  const int sa = s_shift[ea], sb = s_shift[eb], na = s_exp[ea], nb = s_exp[eb];
  const double fa = s_scale[ea], fb = s_scale[eb];
  const uint32_t dbase = (uint32_t)__cvta_generic_to_shared(dig) + lane * 16;
  // level sums of the 8 outputs of a tile of one parity, as integers
  auto sums = [&](int ks0, int ks_n, const uint4* __restrict__ mat, long long (&T)[4]) {
    long long hi[4] = {0, 0, 0, 0}, lo[4] = {0, 0, 0, 0};
    for (int s0 = 0; s0 < ks_n; s0 += TF_SEG) {
      float acc[8][4];
#pragma unroll
      for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[p][i] = 0.f;
      const int s1 = min(s0 + TF_SEG, ks_n);
#pragma unroll 2
      for (int ks = s0; ks < s1; ++ks) {
        uint4 b[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) b[v] = __ldg(mat + (ks * 4 + v) * 32);
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          uint32_t af[4];
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                       : "=r"(af[0]), "=r"(af[1]), "=r"(af[2]), "=r"(af[3])
                       : "r"(dbase + (p * KS + ks0 + ks) * 512));
#pragma unroll
          for (int r = 0; r + p < 8; ++r) {
            const uint4& w = b[r >> 1];
            mma16816(acc[p + r], af, (r & 1) ? w.z : w.x, (r & 1) ? w.w : w.y);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float lev[8] = {acc[0][i], acc[1][i], acc[2][i], acc[3][i], acc[4][i], acc[5][i], acc[6][i], acc[7][i]};
        add_levels(lev, hi[i], lo[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // >> s, rounded
      const int s = i < 2 ? sa : sb;
      T[i] = (hi[i] << (32 - s)) + ((lo[i] + (1ll << (s - 1))) >> s);
    }
  };
  // where the lane's two rows go
  const long la = l0 + row, lb = YM ? la : la + 8;
  const bool oka = la < a.lines, okb = lb < a.lines;
  double* out = a.out[f];
  const uint4 *mat_e = a.mat + lane, *mat_o = mat_e + (size_t)sh.tiles_e * sh.ks_e * 128;
  for (int tile = warp; tile < sh.tiles_e; tile += TF_THREADS / 32) {  // tiles_o <= tiles_e
    __syncwarp();  // lanes without a line left the last tile's stores early; ldmatrix and mma take whole warps
    long long E[4], O[4];
    sums(0, sh.ks_e, mat_e + (size_t)tile * sh.ks_e * 128, E);
    sums(sh.ks_e, tile < sh.tiles_o ? sh.ks_o : 0, mat_o + (size_t)tile * sh.ks_o * 128, O);
    const int n0 = 8 * tile + 2 * cq;
    if constexpr (MODE == TF_Z || MODE == TF_Z2) {
      const size_t ld = 2 * (size_t)d.modes();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int n = n0 + (i & 1), ns = i < 2 ? na : nb;
        const double fs = i < 2 ? fa : fb;
        if (!(i < 2 ? oka : okb)) continue;
        double* o = out + (i < 2 ? la : lb);
        if (MODE == TF_Z2) {
          if (n < sh.n_e) o[(size_t)(2 * n) * ld] = scaled(E[i], ns, fs) * a.scale;
          if (n < sh.n_o) o[(size_t)(2 * n + 1) * ld] = scaled(O[i], ns, fs) * a.scale;
        } else if (n < sh.n_e) {
          o[(size_t)n * ld] = scaled(E[i] + O[i], ns, fs);
          if (sh.L - n > n) o[(size_t)(sh.L - n) * ld] = scaled(E[i] - O[i], ns, fs);
        }
      }
    } else if constexpr (YM) {
      if (!oka) continue;
      const long p = la / d.KX;
      const int kx = (int)(la - p * d.KX);
      double2* o = reinterpret_cast<double2*>(out) + (size_t)p * (MODE == TF_YINV ? d.PY : d.KY) * d.KX + kx;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int n = n0 + i;
        if (n >= sh.n_e) continue;
        const long long er = E[i], ei = E[2 + i], pr = O[i], pi = O[2 + i];
        // E + i O and E - i O
        const double2 plus = make_double2(scaled(er - pi, na, fa), scaled(ei + pr, na, fa));
        const double2 minus = make_double2(scaled(er + pi, na, fa), scaled(ei - pr, na, fa));
        if (MODE == TF_YINV) {
          o[(size_t)n * d.KX] = plus;
          if (n > 0 && 2 * n < sh.L) o[(size_t)(sh.L - n) * d.KX] = minus;
        } else {  // modes 0 .. NYQ in place, the negative ones 1 .. NYQ - 1 from the top
          o[(size_t)n * d.KX] = make_double2(minus.x * a.scale, minus.y * a.scale);
          if (n > 0 && n < d.NYQ) o[(size_t)(d.KY - n) * d.KX] = make_double2(plus.x * a.scale, plus.y * a.scale);
        }
      }
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (!(h ? okb : oka)) continue;
        const double fs = h ? fb : fa;
        const int ns = h ? nb : na;
        const long r = h ? lb : la;
        if (MODE == TF_XINV) {
          double* o = out + (size_t)r * d.PX;
          const double x0 = scaled(E[2 * h] - O[2 * h], ns, fs), x1 = scaled(E[2 * h + 1] - O[2 * h + 1], ns, fs);
          if (n0 + 1 < sh.n_e)
            *reinterpret_cast<double2*>(o + n0) = make_double2(x0, x1);
          else if (n0 < sh.n_e)
            o[n0] = x0;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int n = n0 + i;
            if (n > 0 && 2 * n < sh.L) o[sh.L - n] = scaled(E[2 * h + i] + O[2 * h + i], ns, fs);
          }
        } else {
          double2* o = reinterpret_cast<double2*>(out) + (size_t)r * d.KX;
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (n0 + i < sh.n_e) o[n0 + i] = make_double2(scaled(E[2 * h + i], ns, fs), scaled(-O[2 * h + i], ns, fs));
        }
      }
    }
  }
}

// The Lamb vector at every point of the product grid, in place of the first
// three of the six fields u, v, w, ox, oy, oz:
//   H1 = oy w - re_p - oz v, H2 = oz u - ox w, H3 = ox v - oy u.
// Two points per thread (n is even); bound by memory and the FP64 pipe alike.
__global__ void __launch_bounds__(256) k_lamb64(double* __restrict__ wp, size_t n, double re_p) {
  const size_t i = 2 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= n) return;
  double2 x[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) x[f] = *reinterpret_cast<const double2*>(wp + f * n + i);
  const double2 &u = x[0], &v = x[1], &w = x[2], &ox = x[3], &oy = x[4], &oz = x[5];
  *reinterpret_cast<double2*>(wp + i) =
      make_double2((oy.x * w.x - re_p) - oz.x * v.x, (oy.y * w.y - re_p) - oz.y * v.y);
  *reinterpret_cast<double2*>(wp + n + i) = make_double2(oz.x * u.x - ox.x * w.x, oz.y * u.y - ox.y * w.y);
  *reinterpret_cast<double2*>(wp + 2 * n + i) = make_double2(ox.x * v.x - oy.x * u.x, ox.y * v.y - oy.y * u.y);
}

// Matrix digits in fragment order: [n8 tile][ks][4][lane] uint4, a lane's 16 words holding, per plane, k = 2 (lane % 4), + 1 and the
// same + 8 of output lane / 4.  cosine and sine of 2 pi j / period as
// 62-bit integers (times the transform's factor 2^-f); entry (n, k) is
// table[(n' k') mod period], halved where the transform says.
template <int MODE>
__global__ void k_tf_matrix(const long long* __restrict__ cs, const long long* __restrict__ sn, TfShape s, int period,
                            uint4* __restrict__ out) {
  const int ne = s.tiles_e * s.ks_e, total = ne + s.tiles_o * s.ks_o;  // (tile, ks) items of 32 lanes
  const int item = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
  if (item >= total) return;
  const bool odd = item >= ne;
  const int it = odd ? item - ne : item, ksn = odd ? s.ks_o : s.ks_e;
  const int ks = it % ksn, tile = it / ksn;
  const int n = 8 * tile + lane / 4, kn = odd ? s.k_o : s.k_e, nn = odd ? s.n_o : s.n_e;
  long long x[4];
  for (int i = 0; i < 4; ++i) {
    const int k = 16 * ks + 2 * (lane & 3) + (i & 1) + 8 * (i >> 1);
    x[i] = 0;
    if (k >= kn || n >= nn) continue;
    long long v;  // the doubled modes' tables hold 2^61 cos, sin, the others 2^62
    if (MODE == TF_Z) {
      v = cs[((long)n * (2 * k + (odd ? 1 : 0))) % period];
    } else if (MODE == TF_Z2) {  // 2 cos, halved at the end points and for coefficient 0
      v = cs[((long)(2 * n + (odd ? 1 : 0)) * k) % period] * (k == 0 ? 1 : 2);
      if (n == 0 && !odd) v >>= 1;
    } else {
      v = (odd ? sn : cs)[((long)n * k) % period];
      if (MODE == TF_XINV && k > 0) v *= 2;
    }
    x[i] = v;
  }
  const long long y[8] = {x[0], x[1], x[2], x[3], 0, 0, 0, 0};
  uint32_t w[8][4];  // per plane (k, k + 1) and (k + 8, k + 9) as FP16 pairs
  digit_halves(y, w);
  uint4* o = out + (size_t)item * 128 + lane;
  for (int v = 0; v < 4; ++v) o[v * 32] = make_uint4(w[2 * v][0], w[2 * v][1], w[2 * v + 1][0], w[2 * v + 1][1]);
}

// one * cos, one * sin(2 pi j / L) as integers (L = 2^a 3^b 5^c).  Rounded each
// by itself, the cosines of a whole turn would sum to a few units instead of
// zero, and a line constant in x, y or z would leak that into its other modes
// (an FFT's butterflies cancel it exactly, so laminar flow stays laminar).
// So only independent entries are rounded: of every coset j + t L / p, p prime,
// the one whose component modulo p^e has the top digit p - 1 is minus the sum
// of the others, which makes the sum over every subgroup zero; adding the
// mirror image (of half the size) restores the symmetry.  Entries stay within
// a few units of their values.
void trig_table(int L, long double one, std::vector<long long>& cs, std::vector<long long>& sn) {
  const long double pi2 = 6.283185307179586476925286766559005768L;
  std::vector<long long> t[2];
  for (auto& v : t) v.resize(L);
  for (int j = 0; j <= L / 2; ++j) {
    const long double w = pi2 * j / L;
    const long long c = llrintl(cosl(w) * one * 0.5L), s = llrintl(sinl(w) * one * 0.5L);
    t[0][j] = c;
    t[1][j] = s;
    if (j > 0 && j < L - j) {
      t[0][L - j] = c;
      t[1][L - j] = -s;
    }
  }
  for (int p : {2, 3, 5}) {
    if (L % p) continue;
    int pe = 1;
    while ((L / pe) % p == 0) pe *= p;
    for (auto& v : t)
      for (int j = 0; j < L / p; ++j) {
        long long sum = 0;
        int last = -1;
        for (int q = 0; q < p; ++q) {
          const int i = j + q * (L / p);
          if ((i % pe) / (pe / p) == p - 1) last = i;
          else sum += v[i];
        }
        v[last] = -sum;
      }
  }
  cs.resize(L);
  sn.resize(L);
  for (int j = 0; j < L; ++j) {
    const int m = (L - j) % L;
    cs[j] = t[0][j] + t[0][m];
    sn[j] = t[1][j] - t[1][m];
  }
}

size_t tf_smem(const TfShape& s) { return (size_t)8 * 512 * (s.ks_e + s.ks_o); }
size_t tf_mat_vecs(const TfShape& s) {
  return ((size_t)s.tiles_e * s.ks_e + (size_t)s.tiles_o * s.ks_o) * 128;
}

TfShape tf_shape(int L, int ke, int ko, int ne, int no) {
  TfShape s{};
  s.L = L;
  s.k_e = ke;
  s.k_o = ko;
  s.n_e = ne;
  s.n_o = no;
  s.ks_e = (ke + 15) / 16;
  s.ks_o = (ko + 15) / 16;
  s.tiles_e = (ne + 7) / 8;
  s.tiles_o = (no + 7) / 8;
  return s;
}


template <int MODE>
int launch_tf(Handle* h, const Dims& d, const TfPlan& p, const double* const* in, double* const* out, int nfields,
              long lines, int kid) {  // kid < 0: not one of a step's kernels
  TfArgs a{};
  for (int i = 0; i < nfields; ++i) {
    a.in[i] = in[i];
    a.out[i] = out[i];
  }
  a.nfields = nfields;
  a.scale = MODE == TF_YFWD ? 1.0 / ((double)d.PX * (double)d.PY) : MODE == TF_Z2 ? 1.0 / (double)d.MZ : 1.0;
  a.mat = static_cast<const uint4*>(p.mat);
  a.s = p.s;
  a.lines = lines;
  a.d = d;
  const size_t smem = tf_smem(p.s);
  if (!cuda_ok(h, cudaFuncSetAttribute(k_tf<MODE>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       (int)cudaSharedmemCarveoutMaxShared),
               "k_tf") ||
      !cuda_ok(h, cudaFuncSetAttribute(k_tf<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "k_tf smem"))
    return CHF_E_CUDA;
  const int per = MODE == TF_YINV || MODE == TF_YFWD ? TF_LINES / 2 : TF_LINES;
  cudaEvent_t ev;
  if (kid >= 0) prof_begin(h, kid, &ev);
  k_tf<MODE><<<(unsigned)((lines + per - 1) / per * nfields), TF_THREADS, smem, h->stream>>>(a);
  if (kid >= 0) prof_end(h, kid, ev);
  return cuda_ok(h, cudaGetLastError(), "k_tf") ? CHF_OK : CHF_E_CUDA;
}

// h_v = k^2 H2 + D (i a H1 + i b H3) and h_g = i a H3 - i b H1 (REF:1502-1540)
// from the coefficients H1, H2, H3 [NZ][2 modes], the (0,0) mode carrying H1,
// H3.  One thread per real column and parity chain of the derivative
// recurrence b_k = b_{k+2} + 2 (k + 1) G_{k+1} (dz, REF:570-599), b_0 halved;
// bound by its loads (5 reads and 2 writes of 8 bytes per element).
constexpr int CURL64_THREADS = 64;
constexpr int CURL64_PF = 4;
__global__ void __launch_bounds__(CURL64_THREADS) k_curl64(const double* __restrict__ H1, const double* __restrict__ H2,
                                                         const double* __restrict__ H3, double* __restrict__ hv,
                                                         double* __restrict__ hg, const double* __restrict__ iapha,
                                                         const double* __restrict__ ibeta, Dims d) {
  const long ncols = 2 * d.modes(), col = (long)blockIdx.x * (CURL64_THREADS / 2) + (threadIdx.x & 31);
  const int par = threadIdx.x >> 5, N = d.N;
  if (col >= ncols) return;
  const long m = col >> 1;
  const double a = iapha[m % d.KX], b = ibeta[m / d.KX], k2 = a * a + b * b;
  const double s = (col & 1) ? 1.0 : -1.0;  // (i z)_re = -z_im, (i z)_im = z_re
  const double sa = s * a, sb = s * b;
  const bool mean = m == 0;
  const long pc = mean ? col : (col ^ 1);
  double dg2 = 0.0;
  const int ktop = ((N - par) & ~1) | par;
  for (int k0 = ktop; k0 >= 0; k0 -= 2 * CURL64_PF) {
    double x1[CURL64_PF], x3[CURL64_PF], y1[CURL64_PF], y2[CURL64_PF], y3[CURL64_PF];
#pragma unroll
    for (int i = 0; i < CURL64_PF; ++i) {
      const int k = max(k0 - 2 * i, 0);
      const size_t at = (size_t)k * ncols, up = (size_t)min(k + 1, N) * ncols;
      x1[i] = H1[up + pc];
      x3[i] = H3[up + pc];
      y1[i] = H1[at + pc];
      y3[i] = H3[at + pc];
      y2[i] = H2[at + col];
    }
#pragma unroll
    for (int i = 0; i < CURL64_PF; ++i) {
      const int k = k0 - 2 * i;
      if (k < 0) break;
      double dg = 0.0;
      if (k < N) dg = fma((double)(2 * (k + 1)), fma(sa, x1[i], sb * x3[i]), dg2);
      dg2 = dg;
      if (k == 0) dg *= 0.5;
      hv[(size_t)k * ncols + col] = mean ? y1[i] : fma(k2, y2[i], dg);
      hg[(size_t)k * ncols + col] = mean ? y3[i] : fma(sa, y3[i], -(sb * y1[i]));
    }
  }
}


}  // namespace

// Whether the digit products serve the wall-normal / the in-plane transforms
// of a grid: the dense product's work grows with the square of the line, the
// FFT's hardly.  Measured, digits against FFTs: z on 160, 300 and 500 product
// intervals 0.26 / 1.26, 0.29 / 0.71 and 0.48 / 1.14 ms (the longest that fit
// shared memory by far); x and y on lines of 240, 300, 384 and 480 points
// 1.07 / 1.74, 1.80 / 2.41, 2.99 / 3.33 and 5.16 / 3.91 ms.
// A device without room for their work space (spare_memory) keeps the FFTs.
constexpr int kTfMaxZ = 512, kTfMaxXY = 384;
static bool z_lines(const Dims& d) { return d.nch == 1 && d.MZ <= kTfMaxZ; }
static bool xy_lines(const Dims& d) { return d.nch == 1 && d.PX <= kTfMaxXY && d.PY <= kTfMaxXY; }
bool tf_z(const Handle* h) { return h->tf_image && z_lines(h->d); }
bool tf_xy(const Handle* h) { return h->wp != nullptr; }

// the unpadded lines of the physical velocity: the same lengths (chf_phys.cu has the figures)
bool tf_phys(const Dims& d) { return d.nch == 1 && d.nnx <= kTfMaxXY && d.nny <= kTfMaxXY; }

namespace {

struct TfItem {
  TfPlan* p;
  int mode, period;
};

// the digit matrices of the items' plans, in one allocation.  *image says that
// they are there (setup_tf, setup_tf_out), so it and the plans' pointers are set
// after the last step of the set-up has succeeded; a failed one leaves them null
// and is done again by the next call.
int build_tf(Handle* h, const std::vector<TfItem>& items, void** image) {
  size_t vecs = 0, entries = 0;
  for (const TfItem& it : items) {
    vecs += tf_mat_vecs(it.p->s);
    entries += 2 * (size_t)it.period;
  }
  std::vector<long long> host;
  host.reserve(entries);
  for (const TfItem& it : items) {
    it.p->s.f = it.mode == TF_XINV || it.mode == TF_Z2 ? 1 : 0;
    std::vector<long long> cs, sn;
    trig_table(it.period, ldexpl(1.0L, 62 - it.p->s.f), cs, sn);
    host.insert(host.end(), cs.begin(), cs.end());
    host.insert(host.end(), sn.begin(), sn.end());
  }
  void* mem = nullptr;
  if (!cuda_ok(h, cudaMalloc(&mem, sizeof(uint4) * vecs + sizeof(long long) * entries), "transform digits")) {
    cudaGetLastError();
    return CHF_E_NOMEM;
  }
  uint4* const first = static_cast<uint4*>(mem);
  const long long* tab = reinterpret_cast<const long long*>(first + vecs);
  bool good = cuda_ok(h, cudaMemcpyAsync((void*)tab, host.data(), sizeof(long long) * entries, cudaMemcpyHostToDevice,
                                         h->stream),
                      "transform tables");
  uint4* mat = first;
  for (const TfItem& it : items) {
    if (!good) break;
    const TfShape& s = it.p->s;
    const int blocks = (int)((tf_mat_vecs(s) / 128 + 3) / 4);
    const long long *cs = tab, *sn = tab + it.period;
    if (it.mode == TF_Z) k_tf_matrix<TF_Z><<<blocks, 128, 0, h->stream>>>(cs, sn, s, it.period, mat);
    else if (it.mode == TF_Z2) k_tf_matrix<TF_Z2><<<blocks, 128, 0, h->stream>>>(cs, sn, s, it.period, mat);
    else if (it.mode == TF_XINV) k_tf_matrix<TF_XINV><<<blocks, 128, 0, h->stream>>>(cs, sn, s, it.period, mat);
    else k_tf_matrix<TF_YINV><<<blocks, 128, 0, h->stream>>>(cs, sn, s, it.period, mat);
    good = cuda_ok(h, cudaGetLastError(), "k_tf_matrix");
    mat += tf_mat_vecs(s);
    tab += 2 * it.period;
  }
  good = good && cuda_ok(h, cudaStreamSynchronize(h->stream), "transform tables");
  if (!good) {
    cudaFree(mem);
    cudaGetLastError();  // or the next launch's check would report it again
    return CHF_E_CUDA;
  }
  mat = first;
  for (const TfItem& it : items) {
    it.p->mat = mat;
    mat += tf_mat_vecs(it.p->s);
  }
  *image = mem;
  return CHF_OK;
}

}  // namespace

// CHF_E_NOMEM from build_tf leaves the FFTs in charge too
int setup_tf(Handle* h) {
  const Dims& d = h->d;
  if (h->tf_image) return CHF_OK;
  const bool z = z_lines(d);
  bool xy = xy_lines(d);
  void* wp = nullptr;
  if (xy) {
    const size_t bytes = sizeof(double) * 6 * (size_t)d.MP * d.PY * d.PX;
    xy = spare_memory(h, bytes) && cudaMalloc(&wp, bytes) == cudaSuccess;
    if (!xy) cudaGetLastError();
  }
  if (!z && !xy) return CHF_OK;
  const int M = d.MZ, N = d.N;
  h->tf_z1.s = tf_shape(M, N / 2 + 1, N / 2, M / 2 + 1, (M + 1) / 2);
  h->tf_gl.s = tf_shape(N, N / 2 + 1, N / 2, N / 2 + 1, N / 2);
  h->tf_z2.s = tf_shape(M, M / 2 + 1, (M + 1) / 2, N / 2 + 1, N / 2);
  h->tf_yi.s = tf_shape(d.PY, d.NYQ, d.NYQ, d.PY / 2 + 1, d.PY / 2);
  h->tf_yf.s = tf_shape(d.PY, d.PY / 2 + 1, d.PY / 2, d.NYQ + 1, d.NYQ + 1);
  h->tf_xi.s = tf_shape(d.PX, d.KX, d.KX, d.PX / 2 + 1, d.PX / 2);
  h->tf_xf.s = tf_shape(d.PX, d.PX / 2 + 1, d.PX / 2, d.KX, d.KX);
  const TfItem all[] = {{&h->tf_z1, TF_Z, 2 * M},
                        {&h->tf_gl, TF_Z, 2 * N},
                        {&h->tf_z2, TF_Z2, 2 * M},
                        {&h->tf_yi, TF_YINV, d.PY},
                        {&h->tf_yf, TF_YFWD, d.PY},
                        {&h->tf_xi, TF_XINV, d.PX},
                        {&h->tf_xf, TF_XFWD, d.PX}};
  const int rc = build_tf(h, std::vector<TfItem>(all + (z ? 0 : 3), all + (xy ? 7 : 3)), &h->tf_image);
  if (rc == CHF_OK)
    h->wp = static_cast<double*>(wp);
  else
    cudaFree(wp);
  if (rc != CHF_E_NOMEM) return rc;
  h->err.clear();
  return CHF_OK;
}

// The unpadded transforms of the statistics and the physical velocity: values
// at the Gauss-Lobatto points, and (tf_phys) on the nnx x nny points of a plane.
int setup_tf_out(Handle* h) {
  if (h->tf_out_image) return CHF_OK;
  const Dims& d = h->d;
  h->tf_oz.s = tf_shape(d.N, d.N / 2 + 1, d.N / 2, d.N / 2 + 1, d.N / 2);
  std::vector<TfItem> items{{&h->tf_oz, TF_Z, 2 * d.N}};
  if (tf_phys(d)) {
    h->tf_oy.s = tf_shape(d.nny, d.NYQ, d.NYQ, d.nny / 2 + 1, d.nny / 2);
    h->tf_ox.s = tf_shape(d.nnx, d.KX, d.KX, d.nnx / 2 + 1, d.nnx / 2);
    items.push_back({&h->tf_oy, TF_YINV, d.nny});
    items.push_back({&h->tf_ox, TF_XINV, d.nnx});
  }
  return build_tf(h, items, &h->tf_out_image);
}

// coefficients -> values at the Gauss-Lobatto points, n fields
int launch_tf_gl(Handle* h, const cd* const* in, cd* const* out, int n) {
  const double* i[6];
  double* o[6];
  for (int f = 0; f < n; ++f) {
    i[f] = reinterpret_cast<const double*>(in[f]);
    o[f] = reinterpret_cast<double*>(out[f]);
  }
  return launch_tf<TF_Z>(h, h->d, h->tf_oz, i, o, n, 2 * h->d.modes(), -1);
}

// Gauss-Lobatto values -> the physical nnx x nny planes, each field in place:
// a CTA has its lines in shared memory before it writes the first of them, and
// the unpadded lines take the place they had.
int launch_tf_plane(Handle* h, cd* const* f, int n) {
  Dims d = h->d;
  d.PX = d.nnx;
  d.PY = d.nny;
  double* x[6];
  for (int i = 0; i < n; ++i) x[i] = reinterpret_cast<double*>(f[i]);
  const int rc = launch_tf<TF_YINV>(h, d, h->tf_oy, x, x, n, (long)d.NZ * d.KX, -1);
  return rc != CHF_OK ? rc : launch_tf<TF_XINV>(h, d, h->tf_ox, x, x, n, (long)d.NZ * d.nny, -1);
}

// the six fields' values on the product grid: state -> wz
int launch_tf_c2v(Handle* h) {
  const size_t zf = (size_t)h->d.MP * h->d.modes();
  const int order[6] = {F_U, F_V, F_W, F_OX, F_OY, F_OZ};
  const double* in[6];
  double* out[6];
  for (int i = 0; i < 6; ++i) {
    in[i] = reinterpret_cast<const double*>(h->f[order[i]]);
    out[i] = reinterpret_cast<double*>(h->wz + i * zf);
  }
  return launch_tf<TF_Z>(h, h->d, h->tf_z1, in, out, 6, 2 * h->d.modes(), K_ZC2V);
}

// y and x inverse, products, x and y forward: wz -> wy -> wp -> wy -> wz (three components)
int launch_tf_xy(Handle* h) {
  const Dims& d = h->d;
  const size_t zf = (size_t)d.MP * d.modes(), yf = (size_t)d.MP * d.PY * d.KX, xf = (size_t)d.MP * d.PY * d.PX;
  double *z[6], *y[6], *x[6];
  for (int i = 0; i < 6; ++i) {
    z[i] = reinterpret_cast<double*>(h->wz + i * zf);
    y[i] = reinterpret_cast<double*>(h->wy + i * yf);
    x[i] = h->wp + i * xf;
  }
  const long ylines = (long)d.MP * d.KX, rows = (long)d.MP * d.PY;
  int rc;
  if ((rc = launch_tf<TF_YINV>(h, h->d, h->tf_yi, z, y, 6, ylines, K_YINV)) != CHF_OK ||
      (rc = launch_tf<TF_XINV>(h, h->d, h->tf_xi, y, x, 6, rows, K_XINV)) != CHF_OK)
    return rc;
  cudaEvent_t ev;
  prof_begin(h, K_LAMB64, &ev);
  k_lamb64<<<(unsigned)((xf / 2 + 255) / 256), 256, 0, h->stream>>>(h->wp, xf, h->cfg.re_p);
  prof_end(h, K_LAMB64, ev);
  if (!cuda_ok(h, cudaGetLastError(), "k_lamb64")) return CHF_E_CUDA;
  if ((rc = launch_tf<TF_XFWD>(h, h->d, h->tf_xf, x, y, 3, rows, K_XPROD)) != CHF_OK) return rc;
  return launch_tf<TF_YFWD>(h, h->d, h->tf_yf, y, z, 3, ylines, K_YFWD);
}

// the Lamb vector's coefficients from its three components on the product
// grid: wz -> hc (3 x [NZ][modes], outside the first half of wz)
int launch_tf_v2c(Handle* h, cd* const* hc) {
  const size_t zf = (size_t)h->d.MP * h->d.modes();
  const double* in[6] = {};
  double* out[6] = {};
  for (int i = 0; i < 3; ++i) {
    in[i] = reinterpret_cast<const double*>(h->wz + i * zf);
    out[i] = reinterpret_cast<double*>(hc[i]);
  }
  return launch_tf<TF_Z2>(h, h->d, h->tf_z2, in, out, 3, 2 * h->d.modes(), K_ZFWD);
}

// values of the Lamb vector's components on the product grid (wz) -> histories
// in the unp1 / wnp1 buffers and clamb1n / clamb3n
int launch_tf_curl(Handle* h) {
  const Dims& d = h->d;
  const size_t zf = (size_t)d.MP * d.modes();
  // omega_x <- H1, omega_z <- H3 (the reference leaves them there,
  // REF:1489-1496); H2, h_v and h_g in the upper half of wz
  cd* hc[3] = {h->f[F_OX], h->wz + 3 * zf, h->f[F_OZ]};
  int rc = launch_tf_v2c(h, hc);
  if (rc != CHF_OK) return rc;
  double* hv = reinterpret_cast<double*>(h->wz + 4 * zf);
  double* hg = reinterpret_cast<double*>(h->wz + 5 * zf);
  const long cols = 2 * d.modes();
  cudaEvent_t ev;
  prof_begin(h, K_CURL32, &ev);
  k_curl64<<<(unsigned)((cols + 31) / 32), CURL64_THREADS, 0, h->stream>>>(
      reinterpret_cast<const double*>(hc[0]), reinterpret_cast<const double*>(hc[1]),
      reinterpret_cast<const double*>(hc[2]), hv, hg, h->iapha, h->ibeta, d);
  prof_end(h, K_CURL32, ev);
  if (!cuda_ok(h, cudaGetLastError(), "k_curl64")) return CHF_E_CUDA;
  const double* in[6] = {hv, hg};
  double* out[6] = {reinterpret_cast<double*>(h->f[F_U]), reinterpret_cast<double*>(h->f[F_W])};
  if ((rc = launch_tf<TF_Z>(h, h->d, h->tf_gl, in, out, 2, cols, K_GL64)) != CHF_OK) return rc;
  return launch_meanfix(h);
}

}  // namespace chf
