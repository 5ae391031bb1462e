// vr_lin.cuh -- real transforms of any length as matrix products.
//
// The lengths that are no power of two have no FFT here: their DCT-II/III along
// z and packed real DFT along theta are products with an N x N matrix.  The
// products are summed in index order from tabulated cosines and sines (the
// device's own cospi and sincospi of the reduced argument), one fused
// multiply-add per term, so a result is the bits of the plain direct sum: the
// mixed form stores its fields in float between the kernels, and a change of
// rounding here would be its whole rounding noise (3e-7 of the velocity) a few
// steps later.
//
// A CTA keeps NC = 32 CPL columns (16 when the line is too long for that) x N
// in shared memory.  A warp takes 16 outputs of its columns at a time, a lane
// holding CPL columns x 16 sums: one shared load of the column's value and
// eight 16-byte loads of coefficients, which all lanes share, feed 16 CPL
// multiply-adds.  The coefficients ([group of 16 outputs][step][16]) stream
// from L2 through a two-stage asynchronous ring of each warp's own, and a
// step's words are in registers before the step before it is done (a step's
// loads and products one after the other: 38 us for 33 below).
// What bounds it with CPL = 2 is the latency of those loads at two warps per
// scheduler (the FP64 pipe would take 12 us), with CPL = 1 the shared-memory
// pipe.  48 x 100 x 180 (theta x r x z; us per transform): a sine and a cosine
// per term, one line per CTA, z 756 and theta 272; here 33 and 17.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "vr_internal.cuh"

namespace vr {

// DCT-II scaled 1/(2 N) and DCT-III on columns M apart (REDFT10, REDFT01); the
// packed real DFT [a0, a1, b1, a2, b2, ...] on lines of N contiguous values
// and its inverse
enum LinKind { kLinZFwd = 0, kLinZInv, kLinThFwd, kLinThInv };
__host__ __device__ constexpr bool lin_theta(int kind) { return kind >= kLinThFwd; }
// the inverses start from entry 0, whose coefficient is 1
__host__ __device__ constexpr int lin_first(int kind) { return kind == kLinZInv || kind == kLinThInv; }
inline size_t lin_table_len(int kind, int N) { return (size_t)16 * ((N + 15) / 16) * (N - lin_first(kind)); }

// the coefficient of entry t in output o, without the scale of the forward
// ones (a template so that every source that includes this shares one)
template <int KIND>
__global__ void k_lin_table(double *tab, int N) {
  constexpr int first = lin_first(KIND);
  const int steps = N - first, n = 16 * ((N + 15) / 16) * steps;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int o = e % 16 + 16 * (e / (16 * steps)), t = (e / 16) % steps + first;
    double v = 0.0;
    if (o < N) {
      if (KIND == kLinZFwd) {
        v = cospi((double)(((long long)(2 * t + 1) * o) % (4 * N)) / (2.0 * N));
      } else if (KIND == kLinZInv) {
        v = 2.0 * cospi((double)(((long long)t * (2 * o + 1)) % (4 * N)) / (2.0 * N));
      } else {
        const int slot = KIND == kLinThFwd ? o : t, pos = KIND == kLinThFwd ? t : o, k = (slot + 1) >> 1;
        double sn, cs;
        sincospi(2.0 * (double)(((long long)pos * k) % N) / N, &sn, &cs);
        const bool cosine = slot == 0 || (slot & 1);
        if (KIND == kLinThFwd)
          v = cosine ? cs : -sn;
        else
          v = !cosine ? sn : 2 * k == N ? 0.5 * cs : cs;  // the Nyquist cosine enters once
      }
    }
    tab[e] = v;
  }
}
// (the error of this launch alone: one that is pending on the thread when a
// context or a solver is made is neither reported nor cleared)
inline cudaError_t lin_table(int kind, int N, double *tab, cudaStream_t s) {
  const int grid = (int)std::min<size_t>(1024, (lin_table_len(kind, N) + 255) / 256);
  void (*const kern[])(double *, int) = {k_lin_table<kLinZFwd>, k_lin_table<kLinZInv>, k_lin_table<kLinThFwd>,
                                         k_lin_table<kLinThInv>};
  void *args[] = {&tab, &N};
  return cudaLaunchKernel((const void *)kern[kind], dim3(grid), dim3(256), args, 0, s);
}

struct LinArg {
  const double *in;
  double *out;
  const double *tab;
  int N;
  int M;         // columns (z: also their stride)
  int nr;        // theta inverse: lines of a dph plane
  int ngroups;   // groups of 16 outputs
  int staged;    // theta: the results leave through shared memory
  int pairs;     // z: the columns come two at a time (M even, in aligned)
};

// line L of the theta transforms' output
template <int KIND>
__device__ __forceinline__ size_t lin_line(const LinArg &a, int L) {
  if (KIND != kLinThInv) return (size_t)L * a.N;
  const int j = 1 + L % a.nr, k = 1 + L / a.nr;
  return (size_t)a.N * (j + (size_t)(a.nr + 2) * k);  // dph(:, j, k)
}

constexpr int kLinKC = 16;  // steps per coefficient stage

// row of the tile: the theta form writes it along its lines, one word to a
// row, so an odd length spreads the banks; the z form's rows come in 16-byte
// pieces
__host__ __device__ constexpr int lin_ld(bool theta, int nc) { return theta ? nc + 1 : nc; }

// NCL lanes along the columns, CPL columns per lane, SUB = 32 / NCL output
// groups per warp
template <int KIND, int NCL, int CPL>
__global__ void __launch_bounds__(512) k_lin(const LinArg a) {
  constexpr int NC = NCL * CPL, LD = lin_ld(lin_theta(KIND), NC), SUB = 32 / NCL, KC = kLinKC, first = lin_first(KIND);
  constexpr bool TH = lin_theta(KIND);
  extern __shared__ double sm[];
  const int N = a.N, steps = N - first;
  const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *x = sm;  // [N][LD]
  double *st0 = sm + (((size_t)N * LD + 1) & ~(size_t)1), *st = st0 + (size_t)warp * 2 * SUB * KC * 16;  // stages
  double *so = st0 + (size_t)nw * 2 * SUB * KC * 16;  // theta: [N][LD] results
  const int c0 = blockIdx.x * NC, nc = min(NC, a.M - c0);
  pdl_wait();
  if (!TH) {
    if (a.pairs) {
      for (int e = threadIdx.x; e < N * (NC / 2); e += blockDim.x) {
        const int k = e / (NC / 2), c = 2 * (e % (NC / 2));
        cp_async16(x + (size_t)k * LD + c, c < nc ? a.in + (size_t)a.M * k + c0 + c : a.in, c < nc ? 16u : 0u);
      }
    } else {
      for (int k = warp; k < N; k += nw)
        for (int c = lane; c < NC; c += 32)
          if (c < nc)
            cp_async8(x + (size_t)k * LD + c, a.in + (size_t)a.M * k + c0 + c);
          else
            x[(size_t)k * LD + c] = 0.0;
    }
  } else {
    for (int l = warp; l < NC; l += nw)
      for (int n = lane; n < N; n += 32)
        if (l < nc)
          cp_async8(x + (size_t)n * LD + l, a.in + (size_t)(c0 + l) * N + n);
        else
          x[(size_t)n * LD + l] = 0.0;
  }
  cp_async_wait_all();
  __syncthreads();
  const int sub = lane / NCL, col = lane % NCL;
  // every lane of a warp runs the same number of steps (an absent group's sums are not stored)
  for (int g0 = (blockIdx.y * nw + warp) * SUB; g0 < a.ngroups; g0 += gridDim.y * nw * SUB) {
    const int g = g0 + sub;
    auto stage = [&](int ch) {
#pragma unroll
      for (int u = 0; u < SUB; u++) {
        const int left = g0 + u < a.ngroups ? (steps - ch * KC) * 8 : 0;  // 16-byte pieces left of this group
        const double *src = a.tab + (left > 0 ? ((size_t)(g0 + u) * steps + (size_t)ch * KC) * 16 : 0);
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
      for (int o = 0; o < 16; o++) acc[c][o] = first ? x[col + 32 * c] : 0.0;
    auto coef = [&](const double *p, double (&w)[16]) {
#pragma unroll
      for (int o = 0; o < 8; o++) {
        const double2 v = *reinterpret_cast<const double2 *>(p + 2 * o);
        w[2 * o] = v.x;
        w[2 * o + 1] = v.y;
      }
    };
    const int nch = (steps + KC - 1) / KC;
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
      const int k0 = ch * KC, k1 = min(steps - k0, KC);
      const double *xs = x + col + (size_t)(first + k0) * LD;
      if constexpr (KIND == kLinThInv) {
        // the cosine and sine of a wavenumber are added first, then to the sum
        int k = 0;
#pragma unroll 2
        for (; k + 1 < k1; k += 2) {
          double wc[16], ws[16];
          coef(cf + k * 16, wc);
          coef(cf + (k + 1) * 16, ws);
#pragma unroll
          for (int c = 0; c < CPL; c++) {
            const double u = xs[k * LD + 32 * c], v = xs[(k + 1) * LD + 32 * c];
#pragma unroll
            for (int o = 0; o < 16; o++) acc[c][o] = acc[c][o] + fma(u, wc[o], v * ws[o]);
          }
        }
        if (k < k1) {  // Nyquist
          double wc[16];
          coef(cf + k * 16, wc);
#pragma unroll
          for (int c = 0; c < CPL; c++)
#pragma unroll
            for (int o = 0; o < 16; o++) acc[c][o] = fma(xs[k * LD + 32 * c], wc[o], acc[c][o]);
        }
      } else {
        // the next step's words load during this step's products
        double w[2][16], v[2][CPL];
        auto fetch = [&](int k, int b) {
          coef(cf + k * 16, w[b]);
#pragma unroll
          for (int c = 0; c < CPL; c++) v[b][c] = xs[k * LD + 32 * c];
        };
        auto mul = [&](int b) {
#pragma unroll
          for (int c = 0; c < CPL; c++)
#pragma unroll
            for (int o = 0; o < 16; o++) acc[c][o] = fma(w[b][o], v[b][c], acc[c][o]);
        };
        fetch(0, 0);
        int k = 0;
        for (; k + 1 < k1; k += 2) {
          fetch(k + 1, 1);
          mul(0);
          fetch(min(k + 2, k1 - 1), 0);
          mul(1);
        }
        if (k < k1) mul(0);
      }
      __syncwarp();  // the stage is refilled next
    }
    if (g < a.ngroups) {
#pragma unroll
      for (int c = 0; c < CPL; c++) {
        const int cc = col + 32 * c;
#pragma unroll
        for (int o = 0; o < 16; o++) {
          const int slot = g * 16 + o;
          if (slot >= N) continue;
          double v = acc[c][o];
          if (KIND == kLinZFwd) v = 2.0 * v / (2.0 * N);
          if (KIND == kLinThFwd) v = slot == 0 ? v / N : (slot & 1) ? 2.0 * v / N : -2.0 * v / N;
          if (TH && a.staged)
            so[(size_t)slot * LD + cc] = v;
          else if (cc < nc)
            a.out[TH ? lin_line<KIND>(a, c0 + cc) + slot : (size_t)a.M * slot + c0 + cc] = v;
        }
      }
    }
  }
  if (TH && a.staged) {  // lines are contiguous: out with lanes along them
    __syncthreads();
    for (int l = warp; l < nc; l += nw) {
      double *o = a.out + lin_line<KIND>(a, c0 + l);
      for (int n = lane; n < N; n += 32) o[n] = so[(size_t)n * LD + l];
    }
  }
}

// shared memory of a CTA of nw warps
inline size_t lin_smem(bool theta, int N, int ncl, int cpl, int nw, bool staged) {
  const size_t ld = lin_ld(theta, ncl * cpl), x = ((size_t)N * ld + 1) & ~(size_t)1;
  return sizeof(double) * (x + (size_t)nw * 2 * (32 / ncl) * kLinKC * 16 + (staged ? x : 0));
}
constexpr size_t kLinSmemMax = 225 * 1024;
// longest line a CTA's shared memory holds (16 columns, 4 warps)
inline bool lin_fits(int N) { return lin_smem(true, N, 16, 1, 4, false) <= kLinSmemMax; }

template <int KIND, int NCL, int CPL>
static cudaError_t lin_launch(const LinArg &a, int nw, int gy, cudaStream_t s) {
  constexpr int NC = NCL * CPL;
  const size_t sm = lin_smem(lin_theta(KIND), a.N, NCL, CPL, nw, a.staged != 0);
  cudaError_t e = allow_dyn_smem(k_lin<KIND, NCL, CPL>, sm);
  if (e) return e;
  return launch_pdl(k_lin<KIND, NCL, CPL>, dim3((a.M + NC - 1) / NC, gy), nw * 32, sm, s, a);
}

// One transform of M columns (z: entry k of column c at in[c + M k]; theta:
// line L at in + L N, the inverse into dph of nr rows).  in != out.
// The z form takes two columns per lane, which halves the loads of
// coefficients (the one-column form is bound by them: 80 % of the shared-memory
// pipe), where that leaves every scheduler a warp's 16 outputs of a tile; 16
// columns where 32 of the line do not fit.  Its output groups are split over
// blockIdx.y: four warps of one group each where two such CTAs fit an SM, else
// all the groups one CTA has warps for, and further while SMs would get
// nothing.  The theta form's lines leave through shared memory whole, so one
// CTA takes all groups, by a multiple of four warps (past 726 positions, where
// a second tile does not fit, they leave directly).
// us per transform before (z split only until two CTAs per SM, one column per
// lane below 2 x 64 columns per SM) and so: z of 48 x 100 x 180 44 / 33, of
// 100 x 64 x 200 70 / 61, of 90 x 128 x 288 210 / 158, of 12 x 64 x 320 39 /
// 25; theta of 100 x 64 x 200 45 / 43; a whole axisymmetric direct solve of
// 512 x 1000 427 / 199, of 128 x 300 82 / 55.
template <int KIND>
static cudaError_t lin_run(const double *in, double *out, const double *tab, int N, int M, int nr, int nsm,
                           cudaStream_t s) {
  constexpr bool TH = lin_theta(KIND);
  constexpr int kMaxWarps = 12;
  LinArg a{in, out, tab, N, M, nr, (N + 15) / 16, TH, !(M & 1) && !((uintptr_t)in & 15)};
  auto shape = [&](int ncl, int cpl, int &nw, int &gy) {
    const int sub = 32 / ncl, nb = (M + ncl * cpl - 1) / (ncl * cpl), gw = (a.ngroups + sub - 1) / sub;
    gy = 1;
    if (TH) {
      nw = std::min(kMaxWarps, (gw + 3) / 4 * 4);
    } else {
      gy = (gw + 3) / 4;
      if (2 * (lin_smem(TH, N, ncl, cpl, 4, false) + 1024) > 227 * 1024) gy = (gw + kMaxWarps - 1) / kMaxWarps;
      gy = std::max(gy, std::min(gw, nsm / nb));
      nw = std::max(4, (gw + gy - 1) / gy);
    }
    while (nw > 4 && lin_smem(TH, N, ncl, cpl, nw, a.staged) > kLinSmemMax) nw--;
    return lin_smem(TH, N, ncl, cpl, nw, a.staged) <= kLinSmemMax;
  };
  int nw, gy;
  if constexpr (!TH)
    if ((M + 63) / 64 * a.ngroups >= 4 * nsm && shape(32, 2, nw, gy)) return lin_launch<KIND, 32, 2>(a, nw, gy, s);
  if (shape(32, 1, nw, gy)) return lin_launch<KIND, 32, 1>(a, nw, gy, s);
  if (shape(16, 1, nw, gy)) return lin_launch<KIND, 16, 1>(a, nw, gy, s);
  a.staged = 0;
  if (shape(16, 1, nw, gy)) return lin_launch<KIND, 16, 1>(a, nw, gy, s);
  return cudaErrorNotSupported;
}

}  // namespace vr
