// vr_fold.cuh -- real transforms of any length as folded matrix products.
//
// The lengths that are no power of two (and the powers below 32) have no
// register FFT here.  Their DCT-II/III along z and packed real DFT along theta
// are products with an N x N matrix whose rows are even or odd about the
// middle of the line, so the line is folded first:
//   forward: S_t = x_t + x_{p(t)}, D_t = x_t - x_{p(t)} (p the mirror
//            position); the even rows need S alone, the odd rows D alone;
//   inverse: E_t from the even entries, O_t from the odd ones;
//            x_t = E_t + O_t, x_{p(t)} = E_t - O_t.
// T positions have a sum (the middle and, for theta, position 0 stand alone)
// and N - T a difference: N multiply-adds per output instead of 2 N.
//
// A CTA keeps NC = 32 CPL columns (16 when the line is too long for that) x N
// in shared memory, difference t at row N - 1 - t.  A warp takes 16 outputs
// of its columns at a time, a lane holding CPL columns x 16 sums: one shared
// load of the column's value and eight 16-byte loads of coefficients, which
// all lanes share, feed 16 CPL fused multiply-adds.  The coefficients
// ([group of 16 outputs][step][16], built on the host by fold_tables) stream
// from L2 through a two-stage asynchronous ring of each warp's own.  What
// bounds it is the FP64 pipe with CPL = 2 (12 shared-memory wavefronts per 16
// issue cycles of multiply-adds) and the shared loads with CPL = 1 (10 per 8).
// At 100 x 48 x 180 (us per transform): direct sums with a sine and cosine per
// term, z 756 and theta 272; this form 29 and 12.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "vr_internal.cuh"

namespace vr {

// kFoldZ: DCT-II scaled 1/(2 N) and DCT-III on columns M apart (REDFT10,
// REDFT01); kFoldTh: the packed real DFT [a0, a1, b1, a2, b2, ...] on lines of
// N contiguous values
enum FoldKind { kFoldZ = 0, kFoldTh = 1 };

// sums of a line of length N (the rest, N - T, are differences)
__host__ __device__ inline int fold_sums(int kind, int N) { return kind == kFoldZ ? (N + 1) / 2 : N / 2 + 1; }
__host__ __device__ inline size_t fold_fwd_len(int kind, int N) {
  const int T = fold_sums(kind, N), D = N - T;
  return (size_t)16 * ((T + 15) / 16 * T + (D + 15) / 16 * D);
}
__host__ __device__ inline size_t fold_inv_len(int kind, int N) {
  const int T = fold_sums(kind, N);
  return (size_t)16 * ((T + 7) / 8) * T;
}

// cos(pi m / (2 N)) from the octant of the integer m
inline double fold_cos(long long m, int N) {
  const long long full = 4LL * N;
  m %= full;
  if (m < 0) m += full;
  if (m > 2LL * N) m = full - m;
  const bool neg = m > N;
  if (neg) m = 2LL * N - m;
  if (m == N) return 0.0;
  const double pi = std::acos(-1.0);
  const double v = 2 * m > N ? std::sin(pi * (double)(N - m) / (2.0 * N)) : std::cos(pi * (double)m / (2.0 * N));
  return neg ? -v : v;
}

// the coefficient tables of one length (fwd: fold_fwd_len, inv: fold_inv_len)
inline void fold_tables(int kind, int N, std::vector<double> &fwd, std::vector<double> &inv) {
  const int T = fold_sums(kind, N), D = N - T;
  std::vector<double> c4((size_t)4 * N);
  for (int m = 0; m < 4 * N; m++) c4[m] = fold_cos(m, N);
  auto cs = [&](long long m) { return c4[(size_t)(((m % (4LL * N)) + 4LL * N) % (4LL * N))]; };
  // entry (sum output i, position t), (difference output i, difference t), without the scale
  auto even = [&](long long i, long long t) { return kind == kFoldZ ? cs(2 * i * (2 * t + 1)) : cs(4 * i * t); };
  auto odd = [&](long long i, long long t) {
    return kind == kFoldZ ? cs((2 * i + 1) * (2 * t + 1)) : cs(N - 4 * (i + 1) * (t + 1));
  };
  fwd.assign(fold_fwd_len(kind, N), 0.0);
  inv.assign(fold_inv_len(kind, N), 0.0);
  const int gs = (T + 15) / 16;
  for (int i = 0; i < T; i++) {
    const double sc = (kind == kFoldZ || i == 0) ? 1.0 / N : 2.0 / N;
    for (int t = 0; t < T; t++) fwd[((size_t)(i / 16) * T + t) * 16 + i % 16] = sc * even(i, t);
  }
  for (int i = 0; i < D; i++) {
    const double sc = kind == kFoldZ ? 1.0 / N : 2.0 / N;
    for (int t = 0; t < D; t++)
      fwd[(size_t)gs * T * 16 + ((size_t)(i / 16) * D + t) * 16 + i % 16] = sc * odd(i, t);
  }
  // inverse: output position t of E (8 per group) and O (8 more); for theta
  // the differences start at position 1
  for (int t = 0; t < T; t++)
    for (int i = 0; i < T; i++) {
      double *p = &inv[((size_t)(t / 8) * T + i) * 16 + t % 8];
      if (kind == kFoldZ) {
        p[0] = (i == 0 ? 1.0 : 2.0) * even(i, t);
        if (i < D) p[8] = 2.0 * odd(i, t);
      } else {
        p[0] = (2 * i == N ? 0.5 : 1.0) * even(i, t);  // the Nyquist cosine enters once
        if (i < D) p[8] = t == 0 ? 0.0 : odd(i, t - 1);
      }
    }
}

struct FoldArg {
  const double *in;
  double *out;
  const double *tab;
  int N, T;
  int M;         // columns (z: also their stride)
  int nr;        // theta inverse: lines of a dph plane; 0 when the output is as the input
  int ngroups;   // groups of 16 outputs (inverse: 8 positions, both halves)
  int staged;    // theta: the results leave through shared memory
};

// line L of the theta transforms' output
__device__ __forceinline__ size_t fold_line(const FoldArg &a, int L) {
  if (!a.nr) return (size_t)L * a.N;
  const int j = 1 + L % a.nr, k = 1 + L / a.nr;
  return (size_t)a.N * (j + (size_t)(a.nr + 2) * k);  // dph(:, j, k)
}

constexpr int kFoldKC = 16;  // steps per coefficient stage

// KIND, DIR (+1 forward, -1 inverse); NCL lanes along the columns, CPL columns
// per lane, SUB = 32 / NCL output groups per warp
template <int KIND, int DIR, int NCL, int CPL>
__global__ void __launch_bounds__(512) k_fold(const FoldArg a) {
  constexpr int NC = NCL * CPL, LD = NC + 1, SUB = 32 / NCL, KC = kFoldKC;
  extern __shared__ double sm[];
  const int N = a.N, T = a.T, D = N - T;
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *x = sm;                                                      // [N][LD]
  double *st = sm + (((size_t)N * LD + 1) & ~(size_t)1) + (size_t)warp * 2 * SUB * KC * 16;  // this warp's stages
  const int c0 = blockIdx.x * NC, nc = min(NC, a.M - c0);
  // ---- the columns; the inverse's even entries go to rows 0 .. T - 1, its odd ones from the end
  if (KIND == kFoldZ) {
    for (int k = warp; k < N; k += nw) {
      const int row = DIR > 0 ? k : (k & 1) ? N - 1 - (k >> 1) : k >> 1;
      for (int c = lane; c < NC; c += 32)
        if (c < nc)
          cp_async8(x + (size_t)row * LD + c, a.in + (size_t)a.M * k + c0 + c);
        else
          x[(size_t)row * LD + c] = 0.0;
    }
  } else {
    for (int l = warp; l < NC; l += nw)
      for (int n = lane; n < N; n += 32) {
        const int row = DIR > 0 ? n : n == 0 ? 0 : (n & 1) ? (n + 1) >> 1 : N - (n >> 1);
        if (l < nc)
          cp_async8(x + (size_t)row * LD + l, a.in + (size_t)(c0 + l) * N + n);
        else
          x[(size_t)row * LD + l] = 0.0;
      }
  }
  cp_async_wait_all();
  __syncthreads();
  if (DIR > 0) {
    constexpr int t0 = KIND == kFoldZ ? 0 : 1;  // first position with a mirror
    for (int t = t0 + warp; t < t0 + D; t += nw) {
      double *p = x + (size_t)t * LD, *q = x + (size_t)(KIND == kFoldZ ? N - 1 - t : N - t) * LD;
      for (int c = lane; c < NC; c += 32) {
        const double u = p[c], v = q[c];
        p[c] = u + v;
        q[c] = u - v;
      }
    }
    __syncthreads();
  }
  const int sub = lane / NCL, col = lane % NCL;
  const int gs = (T + 15) / 16;
  double *so = st - (size_t)warp * 2 * SUB * KC * 16 + (size_t)nw * 2 * SUB * KC * 16;  // theta: [N][LD] results
  // every lane of a warp runs the same number of steps (a short or absent group's extra steps are skipped per step)
  for (int g0 = (blockIdx.y * nw + warp) * SUB; g0 < a.ngroups; g0 += gridDim.y * nw * SUB) {
    const int g = g0 + sub;
    // steps and table of a group; the row of step i
    auto steps_of = [&](int q) { return q >= a.ngroups ? 0 : (DIR < 0 || q < gs) ? T : D; };
    auto tab_of = [&](int q) {
      return a.tab + (size_t)16 * ((DIR < 0 || q < gs) ? (size_t)q * T : (size_t)gs * T + (size_t)(q - gs) * D);
    };
    const int mine = steps_of(g);
    const bool dif = DIR > 0 && g >= gs;
    int most = steps_of(g0);
    if (SUB > 1) most = max(most, steps_of(g0 + SUB - 1));
    auto stage = [&](int ch) {
#pragma unroll
      for (int u = 0; u < SUB; u++) {
        const int left = (steps_of(g0 + u) - ch * KC) * 8;  // 16-byte pieces left of this group
        const double *src = left > 0 ? tab_of(g0 + u) + (size_t)ch * KC * 16 : a.tab;
        double *dst = st + (size_t)((ch & 1) * SUB + u) * KC * 16;
#pragma unroll
        for (int e = 0; e < KC * 8 / 32; e++)
          if (lane + 32 * e < left) cp_async16(dst + 2 * (lane + 32 * e), src + 2 * (lane + 32 * e), 16u);
      }
      cp_async_commit();
    };
    double acc[CPL][16];
#pragma unroll
    for (int c = 0; c < CPL; c++)
#pragma unroll
      for (int o = 0; o < 16; o++) acc[c][o] = 0.0;
    const int nch = (most + KC - 1) / KC;
    stage(0);
    for (int ch = 0; ch < nch; ch++) {
      if (ch + 1 < nch) {
        stage(ch + 1);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncwarp();
      const double *cf = st + (size_t)((ch & 1) * SUB + sub) * KC * 16;
      const int k0 = ch * KC, k1 = min(mine - k0, KC);
      const double *xs = x + col + (size_t)(dif ? N - 1 - k0 : k0) * LD;
      const int xstep = dif ? -LD : LD;
      const double *xd = x + col + (size_t)(N - 1 - k0) * LD;  // the inverse's odd entries
#pragma unroll 4
      for (int k = 0; k < k1; k++) {
        double w[16];
#pragma unroll
        for (int o = 0; o < 8; o++) {
          const double2 v = *reinterpret_cast<const double2 *>(cf + k * 16 + 2 * o);
          w[2 * o] = v.x;
          w[2 * o + 1] = v.y;
        }
#pragma unroll
        for (int c = 0; c < CPL; c++) {
          const double v = xs[k * xstep + 32 * c];
          const double d = DIR < 0 ? xd[-k * LD + 32 * c] : v;
#pragma unroll
          for (int o = 0; o < 8; o++) {
            acc[c][o] = fma(w[o], v, acc[c][o]);
            acc[c][8 + o] = fma(w[8 + o], d, acc[c][8 + o]);
          }
        }
      }
      __syncwarp();  // the stage is refilled next
    }
    if (g < a.ngroups) {
#pragma unroll
      for (int c = 0; c < CPL; c++) {
        const int cc = col + 32 * c;
        auto put = [&](int slot, double v) {
          if (KIND == kFoldTh && a.staged)
            so[(size_t)slot * LD + cc] = v;
          else if (cc < nc)
            a.out[KIND == kFoldTh ? fold_line(a, c0 + cc) + slot : (size_t)a.M * slot + c0 + cc] = v;
        };
        if (DIR > 0) {
#pragma unroll
          for (int o = 0; o < 16; o++) {
            const int i = (dif ? g - gs : g) * 16 + o;
            if (i >= (dif ? D : T)) continue;
            if (KIND == kFoldZ)
              put(2 * i + (dif ? 1 : 0), acc[c][o]);
            else
              put(dif ? 2 * i + 2 : i == 0 ? 0 : 2 * i - 1, acc[c][o]);
          }
        } else {
#pragma unroll
          for (int o = 0; o < 8; o++) {
            const int t = g * 8 + o, m = KIND == kFoldZ ? N - 1 - t : N - t;
            if (t >= T) continue;
            put(t, acc[c][o] + acc[c][8 + o]);
            if (m > t && m < N) put(m, acc[c][o] - acc[c][8 + o]);
          }
        }
      }
    }
  }
  if (KIND == kFoldTh && a.staged) {  // lines are contiguous: out with lanes along them
    __syncthreads();
    for (int l = warp; l < nc; l += nw) {
      double *o = a.out + fold_line(a, c0 + l);
      for (int n = lane; n < N; n += 32) o[n] = so[(size_t)n * LD + l];
    }
  }
}

// shared memory of a CTA of nw warps
inline size_t fold_smem(int N, int ncl, int cpl, int nw, bool staged) {
  const size_t ld = (size_t)ncl * cpl + 1, x = ((size_t)N * ld + 1) & ~(size_t)1;
  return sizeof(double) * (x + (size_t)nw * 2 * (32 / ncl) * kFoldKC * 16 + (staged ? x : 0));
}
constexpr size_t kFoldSmemMax = 225 * 1024;
// longest line a CTA's shared memory holds (16 columns, 4 warps)
inline bool fold_fits(int N) { return fold_smem(N, 16, 1, 4, false) <= kFoldSmemMax; }

template <int KIND, int DIR, int NCL, int CPL>
static cudaError_t fold_launch(const FoldArg &a, int nw, int gy, cudaStream_t s) {
  constexpr int NC = NCL * CPL;
  const size_t sm = fold_smem(a.N, NCL, CPL, nw, a.staged != 0);
  cudaError_t e = allow_dyn_smem(k_fold<KIND, DIR, NCL, CPL>, sm);
  if (e) return e;
  k_fold<KIND, DIR, NCL, CPL><<<dim3((a.M + NC - 1) / NC, gy), nw * 32, sm, s>>>(a);
  return cudaGetLastError();
}

// One transform of M columns (z: entry k of column c at in[c + M k]; theta:
// line L at in + L N, the inverse into dph when nr is set).  in != out.
// Columns per CTA: 64 where those CTAs still give every SM two, else 32 (the
// loads of a column pair share their coefficients, but half the CTAs of a
// small grid would leave SMs idle); 16 where 32 columns of the line do not
// fit.  The z form also splits the output groups over blockIdx.y until there
// are two CTAs per SM; the theta form, whose lines leave through shared
// memory whole, does not (past 726 positions, where a second tile does not
// fit, they leave directly).
template <int KIND, int DIR>
static cudaError_t fold_run(const double *in, double *out, const double *tab, int N, int M, int nr, int nsm,
                            cudaStream_t s) {
  const int T = fold_sums(KIND, N), D = N - T;
  FoldArg a{in, out, tab, N, T, M, nr, DIR > 0 ? (T + 15) / 16 + (D + 15) / 16 : (T + 7) / 8, KIND == kFoldTh};
  auto shape = [&](int ncl, int cpl, int &nw, int &gy) {
    const int sub = 32 / ncl, nb = (M + ncl * cpl - 1) / (ncl * cpl), gw = (a.ngroups + sub - 1) / sub;
    gy = KIND == kFoldZ ? std::min(std::max(1, 2 * nsm / nb), (gw + 3) / 4) : 1;
    nw = std::max(4, std::min(12, (gw + gy - 1) / gy));
    while (nw > 4 && fold_smem(N, ncl, cpl, nw, a.staged) > kFoldSmemMax) nw--;
    return fold_smem(N, ncl, cpl, nw, a.staged) <= kFoldSmemMax;
  };
  int nw, gy;
  if ((M + 63) / 64 >= 2 * nsm && shape(32, 2, nw, gy)) return fold_launch<KIND, DIR, 32, 2>(a, nw, gy, s);
  if (shape(32, 1, nw, gy)) return fold_launch<KIND, DIR, 32, 1>(a, nw, gy, s);
  if (shape(16, 1, nw, gy)) return fold_launch<KIND, DIR, 16, 1>(a, nw, gy, s);
  a.staged = 0;
  if (shape(16, 1, nw, gy)) return fold_launch<KIND, DIR, 16, 1>(a, nw, gy, s);
  return cudaErrorNotSupported;
}

}  // namespace vr
