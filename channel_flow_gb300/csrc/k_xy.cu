// k_xy.cu -- the spanwise and streamwise transforms of getnonlinear
// (poiseuilleflow.f90:1051-1181) on shared-memory lines transformed in place.
//
// Same stages, butterflies and twiddles as the two-buffer kernels of
// k_nonlinear.cu (bit-identical results), other storage.  A line's element
// stays where it is read (fft_place_tables): a butterfly overwrites its own
// inputs, so a stage needs one buffer and one barrier, the first stage reads
// its inputs from global memory (the zero padding is never stored) and the
// last one writes its outputs there.  A 576-point line (16 x 9 x 4) passes
// through shared memory two times instead of five.
//
// Lines lie side by side, [place][line].  y: the 16 streamwise modes of a
// tile fill 128 bytes, so the lanes of a half-warp, which differ in the mode
// only, never share a bank.  x: 8 rows fill 64 bytes and two neighbouring
// places one 128-byte line; `slot` swizzles them so that lanes along the row's
// places (the first stage, which reads consecutive modes from global memory)
// and lanes along the rows (all others) both spread over the banks.
//
// What bounds the x kernel is its instructions between barriers: at 384 x 97 x
// 96 it issues in 59% of the cycles with the shared-memory pipe at 70%, and of
// 109 instructions per point and line two thirds were index arithmetic, most
// of it `slot`.  The places' slots now come from two tables in shared memory
// (90 instructions; 293 -> 237 us there, 2264 -> 1822 us at 384 x 193 x 384,
// 165 -> 138 us at 160 x 97 x 120).  More threads per SM at 56 registers spill
// (2076 us at 384 x 193 x 384), and blocks sized to whole passes of the stages
// change nothing (1822).  The y kernels have no swizzle; at 384 x 193 x 384
// they take 765 us for 2.66 GB and 411 us for 1.33 GB, 0.51 and 0.48 of the
// 6763 GB/s of a copy (loads' latency, and issue in 61 and 50% of the cycles).
#include <algorithm>

#include "chf_internal.h"

namespace chf {

namespace {

using C = cf;
constexpr int kLines = 16;  // y: modes per tile (128 bytes)
constexpr int kRows = 8;    // x: rows per group (64 bytes)
constexpr int Y_THREADS = 256;

// A value as if it came back from memory: keeps the compiler from fusing the
// multiplies of one step (a twiddle, a butterfly) with the additions of the
// next, which would round differently from the two-buffer stages.
__device__ __forceinline__ void settle(C& x) { asm("" : "+f"(x.re), "+f"(x.im)); }

template <int SIGN, int R>
__device__ __forceinline__ void bfly(C* v) {
  if constexpr (R == 2) bfly2<float, SIGN>(v);
  if constexpr (R == 3) bfly3<float, SIGN>(v);
  if constexpr (R == 4) bfly4<float, SIGN>(v);
  if constexpr (R == 5) bfly5<float, SIGN>(v);
  if constexpr (R == 8) bfly8<float, SIGN>(v);
  if constexpr (R == 9) bfly9<float, SIGN>(v);
  if constexpr (R == 16) bfly16<float, SIGN>(v);
#pragma unroll
  for (int r = 0; r < R; ++r) settle(v[r]);
}

// a * w (SIGN < 0) or a * conj(w), with the roundings of the two-buffer stages
// spelled out: the compiler may round either product of a part first, and
// chose differently here and there
template <int SIGN>
__device__ __forceinline__ C turn(C a, C w) {
  if (SIGN < 0)
    return C{__fmaf_rn(a.re, w.re, -__fmul_rn(a.im, w.im)), __fmaf_rn(a.im, w.re, __fmul_rn(a.re, w.im))};
  return C{__fmaf_rn(a.re, w.re, __fmul_rn(a.im, w.im)), __fmaf_rn(a.im, w.re, -__fmul_rn(a.re, w.im))};
}

template <int SIGN, int R>
__device__ __forceinline__ void twiddle(C* v, const C* __restrict__ tws, int Ns, int jm) {
  // 32-bit byte offsets from the table's (uniform) address
  const char* __restrict__ t = reinterpret_cast<const char*>(tws);
  unsigned int o = (unsigned int)jm * sizeof(C);
#pragma unroll
  for (int r = 1; r < R; ++r) {
    v[r] = turn<SIGN>(v[r], *reinterpret_cast<const C*>(t + o));
    o += (unsigned int)Ns * sizeof(C);
  }
}

// f.template operator()<R>() for the stage's radix
template <typename F>
__device__ __forceinline__ void by_radix(int R, F&& f) {
  if (R == 4) f.template operator()<4>();
  else if (R == 8) f.template operator()<8>();
  else if (R == 16) f.template operator()<16>();
  else if (R == 9) f.template operator()<9>();
  else if (R == 2) f.template operator()<2>();
  else if (R == 3) f.template operator()<3>();
  else f.template operator()<5>();
}

// One y transform of a tile of kLines modes of np planes (thread = mode
// tid % kLines, butterflies dealt over the rest): load(plane, n) gives
// element n of the thread's line, store(plane, k, x) takes output k.
template <int SIGN, typename Load, typename Store>
__device__ __forceinline__ void y_lines(C* s, int np, bool live, const FftPlan& p,
                                        const C* __restrict__ stab, const unsigned short* __restrict__ rev,
                                        Load&& load, Store&& store) {
  const int c = threadIdx.x % kLines, id = threadIdx.x / kLines, nid = Y_THREADS / kLines;
  const int L = p.L;
  s += c;
  for (int st = 0; st < p.nst; ++st) {
    if (st > 0) __syncthreads();
    const int Ns = p.Ns[st], last = st == p.nst - 1;
    const unsigned int nrm = p.nr_m[st], lom = p.lo_m[st];
    const int nrs = p.nr_s[st], los = p.lo_s[st];
    const C* __restrict__ tws = stab + p.twoff[st];
    if (!live) continue;
    by_radix(p.R[st], [&]<int R>() {
      const int nr = L / R, LO = nr / Ns;
      for (int b = id; b < np * nr; b += nid) {
        const int pl = fft_div(b, nrm, nrs), bb = b - pl * nr;
        const int hi = fft_div(bb, lom, los), lo = bb - hi * LO;
        const int at = hi * R * LO + lo;  // place of the butterfly's digit 0
        C* line = s + (pl * L + at) * kLines;
        C v[R];
        int jm = 0;
        if (st == 0) {
#pragma unroll
          for (int r = 0; r < R; ++r) v[r] = load(pl, at + r * LO);
        } else {
          jm = rev[p.roff[st] + hi];
#pragma unroll
          for (int r = 0; r < R; ++r) v[r] = line[r * LO * kLines];
          twiddle<SIGN, R>(v, tws, Ns, jm);
        }
        bfly<SIGN, R>(v);
        if (last) {
#pragma unroll
          for (int r = 0; r < R; ++r) store(pl, jm + r * Ns, v[r]);
        } else {
#pragma unroll
          for (int r = 0; r < R; ++r) line[r * LO * kLines] = v[r];
        }
      }
    });
  }
}

// y inverse: 3/2 zero-padding and backward DFT; grid (ceil(KX / kLines),
// ceil(MP / pb), 6), pb planes per CTA
template <int CTAS>
__global__ void __launch_bounds__(Y_THREADS, CTAS) k_yinv_ip(const C* __restrict__ wz, C* __restrict__ wy,
                                                       Dims d, int pb, const __grid_constant__ FftPlan py,
                                                       const C* __restrict__ stab,
                                                       const unsigned short* __restrict__ rev) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int p0 = blockIdx.y * pb, kx = blockIdx.x * kLines + threadIdx.x % kLines;
  const long modes = d.modes();
  const C* __restrict__ src = wz + ((size_t)blockIdx.z * d.MP + p0) * modes + kx;
  C* __restrict__ dst = wy + ((size_t)blockIdx.z * d.MP + p0) * (size_t)d.PY * d.KX + kx;
  const int NYQ = d.NYQ, KX = d.KX, top = d.PY - NYQ, cut = d.PY - d.KY;
  const size_t pstride = (size_t)d.PY * KX;
  y_lines<+1>(
      reinterpret_cast<C*>(smem_raw), min(pb, d.MP - p0), kx < KX, py, stab, rev,
      [&](int pl, int n) {  // the spanwise Nyquist mode is dropped (expand(1))
        const int ky = n < NYQ ? n : n - cut;
        return n < NYQ || n > top ? src[pl * modes + (size_t)ky * KX] : C{(float)0, (float)0};
      },
      [&](int pl, int k, const C& x) { dst[pl * pstride + (size_t)k * KX] = x; });
}

// y forward: forward DFT, truncation (the Nyquist slot takes padded mode
// +NYQ, expand(-1)), 1/(PX PY); grid (ceil(KX / kLines), ceil(MP / pb), 3)
template <int CTAS>
__global__ void __launch_bounds__(Y_THREADS, CTAS) k_yfwd_ip(const C* __restrict__ wy, C* __restrict__ wz,
                                                       Dims d, int pb, const __grid_constant__ FftPlan py,
                                                       const C* __restrict__ stab,
                                                       const unsigned short* __restrict__ rev, float scale) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int p0 = blockIdx.y * pb, kx = blockIdx.x * kLines + threadIdx.x % kLines;
  const long modes = d.modes();
  const C* __restrict__ src = wy + ((size_t)blockIdx.z * d.MP + p0) * (size_t)d.PY * d.KX + kx;
  C* __restrict__ dst = wz + ((size_t)blockIdx.z * d.MP + p0) * modes + kx;
  const int NYQ = d.NYQ, KX = d.KX, top = d.PY - NYQ, cut = d.PY - d.KY;
  const size_t pstride = (size_t)d.PY * KX;
  y_lines<-1>(
      reinterpret_cast<C*>(smem_raw), min(pb, d.MP - p0), kx < KX, py, stab, rev,
      [&](int pl, int n) { return src[pl * pstride + (size_t)n * KX]; },
      [&](int pl, int k, const C& x) {
        if (k <= NYQ || k > top)
          dst[pl * modes + (size_t)(k <= NYQ ? k : k - cut) * KX] = C{x.re * scale, x.im * scale};
      });
}

// Element of row `row` at place `at` of an x line group.  Every part of it is
// an exclusive or of bits of `at` and `row`, so that slot(at, row) is
// slot(at, 0) ^ row, and slot(a + b, row) is slot(a, row) ^ slot(b, 0) where a
// and b have no bit in common.
__device__ __forceinline__ int slot(int at, int row, int swz) {
  constexpr int RB = kRows;
  return (at >> 1) * (2 * RB) + ((at ^ (at >> swz)) & 1) * RB + (row ^ ((at >> 1) & (RB - 1)));
}

// the place of a value of slot(at, 0) (swz >= 1)
__device__ __forceinline__ int place_of(int q, int swz) {
  const int h = q >> 4;
  return 2 * h + (((q >> 3) ^ (h >> (swz - 1))) & 1);
}

// x: c2r of three field pairs, the Lamb products, r2c of (H1 + i H2) and H3;
// rows r = plane * PY + yp as in k_xprod.  ng groups of kRows rows per CTA,
// grid ceil(nrows / (ng kRows)).  The products stand at the inverse
// transform's places, so the forward one works at place[natural index].
template <int THREADS, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS) k_xprod_ip(C* __restrict__ wy, Dims d, float re_p, int ng,
                                                        const __grid_constant__ FftPlan px,
                                                        const C* __restrict__ stab,
                                                        const unsigned short* __restrict__ tab) {
  constexpr int RB = kRows;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* s = reinterpret_cast<C*>(smem_raw);
  const int PX = d.PX, KX = d.KX, L = PX, swz = px.swz, tid = threadIdx.x;
  const long nrows = (long)d.MP * d.PY, r0 = (long)blockIdx.x * ng * RB;
  const size_t fstride = (size_t)d.MP * d.PY * KX;
  const int gl = L * RB;  // elements of one (group, pair) line set, at (g * 3 + pair) * gl
  const int nst = px.nst;
  // the index tables in shared memory (read from the second stage on; the
  // first computes its slots, so as not to wait for them): cold misses on them
  // would otherwise line up behind one another in every CTA, and a slot costs
  // seven instructions where a table read and an exclusive or cost three
  unsigned short* rev = reinterpret_cast<unsigned short*>(s + ng * 3 * gl);
  unsigned short *at_slot = rev + L, *nat_slot = at_slot + L;  // slot(at, 0), slot(place[n], 0)
  for (int t = tid; t < L; t += blockDim.x) {
    rev[t] = tab[t];
    at_slot[t] = (unsigned short)slot(t, 0, swz);
    nat_slot[t] = (unsigned short)slot(tab[L + t], 0, swz);
  }
  // ---- inverse, first stage: lanes along the butterflies of a row
  by_radix(px.R[0], [&]<int R>() {
    const int nr = L / R;
    for (int t = tid; t < ng * 3 * RB * nr; t += blockDim.x) {
      const int lr = fft_div(t, px.nr_m[0], px.nr_s[0]), j = t - lr * nr;
      const int row = lr % RB, gc = lr / RB, g = gc / 3, c = gc - 3 * g;
      const long r = r0 + g * RB + row;
      const C* __restrict__ Fr = wy + (size_t)(2 * c) * fstride + (size_t)r * KX;
      const C* __restrict__ Gr = Fr + fstride;
      const int kend = r < nrows ? KX : 0;
      C v[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int n = j + i * nr, k = min(n, PX - n);
        v[i] = C{(float)0, (float)0};
        if (k < kend) {
          const C F = Fr[k], G = Gr[k];
          // F + i G, its conjugate partner (products by 1 or -1: exact), or
          // the streamwise means (real parts)
          const float u = n < KX ? 1.f : -1.f;
          v[i] = C{__fmaf_rn(-u, G.im, F.re), __fmaf_rn(u, F.im, G.re)};
          if (i == 0 && n == 0) v[i] = C{F.re, G.re};
        }
      }
      bfly<+1, R>(v);
      C* lines = s + gc * gl;
#pragma unroll
      for (int i = 0; i < R; ++i) lines[slot(i * nr + j, row, swz)] = v[i];
    }
  });
  const int row = tid % RB, id = tid / RB, nid = blockDim.x / RB;
  // ---- inverse, middle stages, and the last one when its three butterflies
  // of a place do not fit the registers (radix above 5)
  const int rl = px.R[nst - 1];
  const bool fuse = rl <= 5 && nst > 1;
  for (int st = 1; st < nst - (fuse ? 1 : 0); ++st) {
    __syncthreads();
    by_radix(px.R[st], [&]<int R>() {
      const int Ns = px.Ns[st], nr = L / R, LO = nr / Ns;
      const C* __restrict__ tws = stab + px.twoff[st];
      for (int b = id; b < ng * 3 * nr; b += nid) {
        const int gc = fft_div(b, px.nr_m[st], px.nr_s[st]), bb = b - gc * nr;
        const int hi = fft_div(bb, px.lo_m[st], px.lo_s[st]), at = hi * R * LO + bb - hi * LO;
        C* lines = s + gc * gl;
        C v[R];
        int q[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
          q[i] = at_slot[at + i * LO] ^ row;
          v[i] = lines[q[i]];
        }
        twiddle<+1, R>(v, tws, Ns, rev[px.roff[st] + hi]);
        bfly<+1, R>(v);
#pragma unroll
        for (int i = 0; i < R; ++i) lines[q[i]] = v[i];
      }
    });
  }
  __syncthreads();
  // ---- products: H1 + i H2 in place of pair 0 (u, v), H3 in place of pair 1 (w, ox)
  auto products = [&](const C& a, const C& b, const C& c, C& z1, C& z2) {
    const float u = a.re, v = a.im, w = b.re, ox = b.im, oy = c.re, oz = c.im;
    const float h1 = (oy * w - re_p) - oz * v;
    const float h2 = oz * u - ox * w;
    const float h3 = ox * v - oy * u;
    z1 = C{h1, h2};
    z2 = C{h3, (float)0};
  };
  if (fuse) {
    by_radix(rl, [&]<int R>() {
      if constexpr (R <= 5) {
        const int st = nst - 1, Ns = px.Ns[st];
        const C* __restrict__ tws = stab + px.twoff[st];
        for (int b = id; b < ng * Ns; b += nid) {
          const int g = fft_div(b, px.nr_m[st], px.nr_s[st]), hi = b - g * Ns;
          const int jm = rev[px.roff[st] + hi];
          int q[R];
#pragma unroll
          for (int i = 0; i < R; ++i) q[i] = at_slot[hi * R + i] ^ row;
          C v[3][R];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const C* lines = s + (g * 3 + c) * gl;
#pragma unroll
            for (int i = 0; i < R; ++i) v[c][i] = lines[q[i]];
            twiddle<+1, R>(v[c], tws, Ns, jm);
            bfly<+1, R>(v[c]);
          }
          C* lines = s + g * 3 * gl;
#pragma unroll
          for (int i = 0; i < R; ++i) {
            C z1, z2;
            products(v[0][i], v[1][i], v[2][i], z1, z2);
            lines[q[i]] = z1;
            lines[gl + q[i]] = z2;
          }
        }
      }
    });
  } else {
    for (int b = id; b < ng * L; b += nid) {
      const int g = b / L;
      C* lines = s + g * 3 * gl + (at_slot[b - g * L] ^ row);
      C z1, z2;
      products(lines[0], lines[gl], lines[2 * gl], z1, z2);
      lines[0] = z1;
      lines[gl] = z2;
    }
  }
  // ---- forward stages of the two lines, at place[natural index]
  for (int st = 0; st < nst - (fuse ? 1 : 0); ++st) {
    __syncthreads();
    by_radix(px.R[st], [&]<int R>() {
      const int Ns = px.Ns[st], nr = L / R, LO = nr / Ns;
      const C* __restrict__ tws = stab + px.twoff[st];
      for (int b = id; b < ng * 2 * nr; b += nid) {
        const int gc = fft_div(b, px.nr_m[st], px.nr_s[st]), bb = b - gc * nr;
        const int hi = fft_div(bb, px.lo_m[st], px.lo_s[st]), at = hi * R * LO + bb - hi * LO;
        C* lines = s + ((gc >> 1) * 3 + (gc & 1)) * gl;
        C v[R];
        int q[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
          q[i] = nat_slot[at + i * LO] ^ row;
          v[i] = lines[q[i]];
        }
        if (st > 0) twiddle<-1, R>(v, tws, Ns, rev[px.roff[st] + hi]);
        bfly<-1, R>(v);
#pragma unroll
        for (int i = 0; i < R; ++i) lines[q[i]] = v[i];
      }
    });
  }
  __syncthreads();
  // ---- outputs: H1, H2 from Z[k] and conj Z[-k], H3 directly
  auto emit = [&](long r, int k, const C& A, C B, const C& H3) {
    B.im = -B.im;
    wy[(size_t)r * KX + k] = C{(float)0.5 * (A.re + B.re), (float)0.5 * (A.im + B.im)};
    wy[fstride + (size_t)r * KX + k] = C{(float)0.5 * (A.im - B.im), (float)-0.5 * (A.re - B.re)};
    wy[2 * fstride + (size_t)r * KX + k] = H3;
  };
  if (fuse) {
    // butterflies jm and Ns - jm hold each other's Z[-k]; 0 and (Ns even)
    // Ns / 2 hold their own and share a task
    by_radix(rl, [&]<int R>() {
      if constexpr (R <= 5) {
        const int st = nst - 1, Ns = px.Ns[st], half = (Ns + 1) / 2;
        const C* __restrict__ tws = stab + px.twoff[st];
        for (int b = id; b < ng * half; b += nid) {
          const int g = b / half, jm = b - g * half, jn = jm > 0 ? Ns - jm : Ns % 2 ? 0 : Ns / 2;
          const long r = r0 + g * RB + row;
          C z[2][R], h[2][R];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = e ? jn : jm, at = place_of(nat_slot[j], swz);
            const C* lines = s + g * 3 * gl;
#pragma unroll
            for (int i = 0; i < R; ++i) {
              const int q = nat_slot[at + i] ^ row;
              z[e][i] = lines[q];
              h[e][i] = lines[gl + q];
            }
            twiddle<-1, R>(z[e], tws, Ns, j);
            bfly<-1, R>(z[e]);
            twiddle<-1, R>(h[e], tws, Ns, j);
            bfly<-1, R>(h[e]);
          }
          if (r >= nrows) continue;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (e == 1 && jn == jm) break;
#pragma unroll
            for (int i = 0; i < R; ++i) {
              const int k = (e ? jn : jm) + i * Ns;
              if (k >= KX) continue;
              const C B = jm > 0 ? z[1 - e][R - 1 - i] : e ? z[1][R - 1 - i] : z[0][(R - i) % R];
              emit(r, k, z[e][i], B, h[e][i]);
            }
          }
        }
      }
    });
  } else {
    for (int b = id; b < ng * KX; b += nid) {
      const int g = b / KX, k = b - g * KX;
      const long r = r0 + g * RB + row;
      if (r >= nrows) continue;
      const C* lines = s + g * 3 * gl;
      const int q = nat_slot[place_of(nat_slot[k], swz)] ^ row;
      const int qn = nat_slot[place_of(nat_slot[k == 0 ? 0 : PX - k], swz)] ^ row;
      emit(r, k, lines[q], lines[qn], lines[gl + q]);
    }
  }
}

constexpr size_t kMaxSmem = 227 * 1024;

template <typename K>
bool set_smem(Handle* h, K kernel, size_t bytes) {
  return cuda_ok(h, cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (int)cudaSharedmemCarveoutMaxShared),
                 "cudaFuncSetAttribute") &&
         (bytes <= 48 * 1024 ||
          cuda_ok(h, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes),
                  "cudaFuncSetAttribute"));
}

// sets per CTA so that the first stage gives every thread a butterfly, while
// four CTAs still share an SM and every SM still gets two of the CTAs
int pack(size_t set_bytes, int set_tasks, long sets, int threads, long ctas) {
  int n = 1;
  while (n * set_tasks < threads && n < sets && (n + 1) * set_bytes <= kMaxSmem / 4 && ctas / (n + 1) >= 2) ++n;
  return n;
}

constexpr size_t kSmSmem = 228 * 1024;  // shared memory of an SM; a CTA takes 1 KB more than it asks for

}  // namespace

// Whether the in-place kernels serve these lines: they hold whole tiles of
// lines per CTA (y 128 L bytes, x 198 L bytes).
bool xy_in_place(const Dims& d) { return 128 * (size_t)d.PY <= kMaxSmem && 198 * (size_t)d.PX <= kMaxSmem; }

int launch_y_in_place(Handle* h, cf* wz, cf* wy, const FftPlan& py, const cf* stab, const unsigned short* rev,
                      bool inverse) {
  const Dims d = fft_view(h->d);
  const size_t set = 128 * (size_t)d.PY;
  const int tiles = (d.KX + kLines - 1) / kLines, nf = inverse ? 6 : 3;
  const int pb = pack(set, py.L / py.R[0] * kLines, d.MP, Y_THREADS, (long)d.MP * tiles * nf / h->num_sms);
  dim3 grid(tiles, (d.MP + pb - 1) / pb, nf);
  // four CTAs per SM (64 registers a thread) where their tiles fit, three otherwise
  const bool four = 4 * pb * set <= kMaxSmem;
  auto inv = four ? k_yinv_ip<4> : k_yinv_ip<3>;
  auto fwd = four ? k_yfwd_ip<4> : k_yfwd_ip<3>;
  cudaEvent_t ev;
  if (!(inverse ? set_smem(h, inv, pb * set) : set_smem(h, fwd, pb * set))) return CHF_E_CUDA;
  prof_begin(h, inverse ? K_YINV : K_YFWD, &ev);
  if (inverse)
    inv<<<grid, Y_THREADS, pb * set, h->stream>>>(wz, wy, d, pb, py, stab, rev);
  else
    fwd<<<grid, Y_THREADS, pb * set, h->stream>>>(wy, wz, d, pb, py, stab, rev,
                                                  (float)(1.0 / ((double)d.PX * (double)d.PY)));
  prof_end(h, inverse ? K_YINV : K_YFWD, ev);
  return cuda_ok(h, cudaGetLastError(), "y transform") ? CHF_OK : CHF_E_CUDA;
}

int launch_x_in_place(Handle* h, cf* wy, const FftPlan& px, const cf* stab, const unsigned short* tab) {
  const Dims d = fft_view(h->d);
  const long nrows = (long)d.MP * d.PY;
  const size_t set = 192 * (size_t)d.PX, tables = 6 * (size_t)d.PX;
  // 1024 threads per SM either way: four small CTAs where their lines fit
  const bool small = 4 * (set + tables + 1024) <= kSmSmem;
  const int threads = small ? 256 : 512;
  const int ng = pack(set, 3 * kRows * (px.L / px.R[0]), (nrows + kRows - 1) / kRows, threads,
                      nrows / kRows / h->num_sms);
  const long per = (long)ng * kRows;
  auto kern = small ? k_xprod_ip<256, 4> : k_xprod_ip<512, 2>;
  cudaEvent_t ev;
  if (!set_smem(h, kern, ng * set + tables)) return CHF_E_CUDA;
  prof_begin(h, K_XPROD, &ev);
  kern<<<(unsigned)((nrows + per - 1) / per), threads, ng * set + tables, h->stream>>>(wy, d, (float)h->cfg.re_p, ng,
                                                                                       px, stab, tab);
  prof_end(h, K_XPROD, ev);
  return cuda_ok(h, cudaGetLastError(), "x transform") ? CHF_OK : CHF_E_CUDA;
}

}  // namespace chf
