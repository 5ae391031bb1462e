// vr_tridiag.cu -- the stand-alone tridiagonal solvers of the reference's
// surface: solve_lap_thom (tripar.F90:120-145, trithom.F90:6-29) and
// solve_lap_bthom (btrithom.F90:5-71), batched over independent systems.
// Host arrays in, host arrays out; the device copies are made per call.
#include <cuda_runtime.h>

#include <atomic>
#include <vector>

#include "vr_internal.cuh"

namespace vr {

// Batched Thomas solve (beta(k) = bb(k) - cc(k-1)*aa(k)/beta(k-1),
// gamm(k) = (rhs(k) - aa(k) gamm(k-1)) / beta(k), sol(k) = gamm(k) -
// cc(k)/beta(k) sol(k+1)) of S systems per CTA.
//
// A system is a chain of n dependent steps, so the time is the chain's
// latency and not its bytes: 10.5 MB at 257 x 1024 would take 1.6 us, a
// division per step alone 10 us.  The chain is therefore taken apart:
// - beta is carried as a ratio u(k) / u(k-1) of the leading minors,
//   u(k) = bb(k) u(k-1) - cc(k-1) aa(k) u(k-2), one fused multiply-add per
//   step on the critical path and no division.  The pair is scaled by the
//   power of two of u(k-1) (exact) before each step, so that u(k) is about
//   beta(k): the numbers formed are those of the recurrence above, in range
//   where its are.  The rounding error of u(k) goes along, to be taken out of
//   the ratio where it divides; the next step continues from the rounded one,
//   as the recurrence does.
// - the divisions 1 / beta(k) of a tile are independent of each other and run
//   on all lanes of kThomDiv warps of their own, to twice the precision (ib + lo),
//   so that a multiplication by them rounds once, as a division would.
// - three warps work on three consecutive tiles of KT positions at a time:
//   the minors of one, the divisions of the one before, gamm of the one
//   before that, while a fourth brings the next tile from memory (8-byte
//   asynchronous copies, lanes along a system: full sectors) and stores the
//   tile that is done.  cc/beta goes to the gamm scratch and gamm to sol; the
//   back substitution streams both backwards the same way.
// The positions past n of the last tile, and systems past nbatch, are rows of
// the identity.  aa(1) and cc(n) are not used: they are taken as 0.
//
// A system with a pivot beyond 2^+-480 (inside, a product cc aa that loses bits
// is far below the rounding of u(k)), a cc / beta that is not 0 but below
// 2^-960, infinities or NaN is solved again by the plain recurrence
// (thomas_plain), one thread per system: 275 us at 257 x 1024 if all are such.
//
// 257 x 1024 (us per call): one thread per system with its loads a system
// apart 241; this form 18.4, with one dividing warp 22.5.  Error against 64
// bits there, of the largest entry: recurrence 1.1e-16, here 9.6e-17 (a
// multiplication by the rounded 1 / beta of the rounded minors: 1.2e-16).
constexpr int kThomKT = 16;    // positions per tile
constexpr int kThomRing = 6;   // tiles in flight
constexpr int kThomArr = 6;    // arrays of a tile
constexpr int kThomDiv = 4;    // warps that divide
constexpr int kThomThreads = 32 * (3 + kThomDiv);

__device__ __forceinline__ int exp_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
// 2^-e of x = m 2^e, 1 <= |m| < 2, for |x| below 2^1023
__device__ __forceinline__ double pow2_inv(double x) {
  return __hiloint2double(0x7fe00000 - (__double2hiint(x) & 0x7ff00000), 0);
}
// whether |x| lies outside 2^-E .. 2^E (0, infinities and NaN do)
template <int E>
__device__ __forceinline__ bool off_range(double x) {
  return 2u * (unsigned)__double2hiint(x) - ((1023u - E) << 21) > (2u * E) << 21;
}
// the exponent by which a factor is scaled, -1022 .. 1022 (0 for infinities and NaN)
__device__ __forceinline__ int scale_exp(double x) {
  const int e = exp_field(x);
  return e == 0x7ff ? 0 : min(max(e - 1023, -1022), 1022);
}
__device__ __forceinline__ double scaled(double x, int e) { return x * __hiloint2double((1023 - e) << 20, 0); }

// x y / d without overflow or underflow on the way
__device__ __forceinline__ double mul_div(double x, double y, double d) {
  const int ex = scale_exp(x), ey = scale_exp(y), ed = scale_exp(d);
  return scalbn(scaled(x, ex) * scaled(y, ey) / scaled(d, ed), ex + ey - ed);
}

// One system by the recurrence as it stands, for any scale of its rows: beta
// is kept in sol until the substitution overwrites it, gamm in its scratch.
__device__ __noinline__ void thomas_plain(const double *r, double *sol, const double *a, const double *d,
                                          const double *c, double *gm, int n) {
  double beta = d[0], g = r[0] / beta;
  sol[0] = beta;
  gm[0] = g;
  for (int k = 1; k < n; k++) {
    beta = d[k] - mul_div(c[k - 1], a[k], beta);
    const int e = max(scale_exp(beta), scale_exp(a[k]));
    g = fma(-scaled(a[k], e), g, scaled(r[k], e)) / scaled(beta, e);
    sol[k] = beta;
    gm[k] = g;
  }
  double x = g;
  sol[n - 1] = x;
  for (int k = n - 2; k >= 0; k--) {
    x = gm[k] - mul_div(c[k], x, sol[k]);
    sol[k] = x;
  }
}

template <int S>
__global__ void __launch_bounds__(kThomThreads) k_thomas(const double *__restrict__ rhs, double *sol,
                                              const double *__restrict__ aa, const double *__restrict__ bb,
                                              const double *__restrict__ cc, double *gamm, int n, int nbatch) {
  constexpr int KT = kThomKT, LD = S + 1, AR = KT * LD, R = kThomRing;
  // arrays of a tile: rhs then gamm, aa, bb then u(k) then 1/beta, cc then cc/beta, u(k-1), the error of u(k) then
  // that of 1/beta
  constexpr int TR = 0, TA = 1, TB = 2, TC = 3, TX = 4, TE = 5;
  extern __shared__ double sm[];
  __shared__ unsigned again;  // systems for thomas_plain
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s0 = blockIdx.x * S, ns = min(S, nbatch - s0);
  const int nt = (n + KT - 1) / KT;
  auto tile = [&](int t, int arr) { return sm + ((size_t)(t % R) * kThomArr + arr) * AR; };
  const size_t base = (size_t)s0 * n;
  double x = 1.0, y = 0.0, cprev = 0.0;  // warp 1: u(k-1), u(k-2) by the scale of u(k-1), cc(k-1)
  double g = 0.0;                        // warp 2: gamm(k-1)
  bool bad = false;                      // of system lane % S
  if (threadIdx.x == 0) again = 0;
  for (int i = 0; i < nt + 5; i++) {
    if (warp == 0) {
      if (i < nt) {
        double *r = tile(i, TR), *a = tile(i, TA), *b = tile(i, TB), *c = tile(i, TC);
#pragma unroll
        for (int e = lane; e < KT * S; e += 32) {
          const int kk = e % KT, s = e / KT, k = i * KT + kk, o = kk * LD + s;
          const size_t q = base + (size_t)s * n + k;
          if (s < ns && k < n) {
            cp_async8(r + o, rhs + q);
            cp_async8(b + o, bb + q);
            if (k > 0) cp_async8(a + o, aa + q); else a[o] = 0.0;
            if (k < n - 1) cp_async8(c + o, cc + q); else c[o] = 0.0;
          } else {
            r[o] = 0.0;
            a[o] = 0.0;
            b[o] = 1.0;
            c[o] = 0.0;
          }
        }
      }
      cp_async_commit();
      const int t = i - 5;  // this tile is done: cc/beta and gamm to memory
      if (t >= 0) {
        const double *f = tile(t, TC), *gm = tile(t, TR);
#pragma unroll
        for (int e = lane; e < KT * S; e += 32) {
          const int kk = e % KT, s = e / KT, k = t * KT + kk;
          const size_t q = base + (size_t)s * n + k;
          if (s < ns && k < n) {
            gamm[q] = f[kk * LD + s];
            sol[q] = gm[kk * LD + s];
          }
        }
      }
      cp_async_wait<1>();  // tile i - 1 has landed
    } else if (warp == 1) {
      const int t = i - 2;
      if (t >= 0 && t < nt && lane < S) {
        const double *a = tile(t, TA) + lane, *c = tile(t, TC) + lane;
        double *b = tile(t, TB) + lane, *xo = tile(t, TX) + lane, *eo = tile(t, TE) + lane;
#pragma unroll
        for (int kk = 0; kk < KT; kk++) {
          const double ak = a[kk * LD], bk = b[kk * LD], p = cprev * ak;
          cprev = c[kk * LD];
          const double s = pow2_inv(x), v = (p * y) * s;
          y = x * s;
          x = fma(bk, y, -v);
          bad |= off_range<480>(x);
          b[kk * LD] = x;
          xo[kk * LD] = y;
          eo[kk * LD] = fma(bk, y, -x) - v;
        }
      }
    } else if (warp >= 3) {
      const int t = i - 3;
      if (t >= 0 && t < nt) {
        double *b = tile(t, TB), *c = tile(t, TC), *eo = tile(t, TE);
        const double *xo = tile(t, TX);
#pragma unroll
        for (int e = threadIdx.x - 96; e < KT * S; e += 32 * kThomDiv) {
          const int o = (e / S) * LD + e % S;
          // 1 / beta = ib + lo of beta = (u(k) + its error) / u(k-1); the last
          // factor, 1 / u(k-1) of a number in [1, 2), needs few bits
          const double u = xo[o], z = b[o], ib = u / z;
          const double lo = (fma(-z, ib, u) - ib * eo[o]) * ib * (double)__frcp_rn((float)u);
          const double ck = c[o], f0 = ck * ib, f = f0 + fma(ck, lo, fma(ck, ib, -f0));
          bad |= off_range<960>(f) && ck != 0.0;
          b[o] = ib;
          eo[o] = lo;
          c[o] = f;
        }
      }
    } else {
      const int t = i - 4;
      if (t >= 0 && t < nt && lane < S) {
        const double *a = tile(t, TA) + lane, *ib = tile(t, TB) + lane, *lo = tile(t, TE) + lane;
        double *r = tile(t, TR) + lane;
#pragma unroll
        for (int kk = 0; kk < KT; kk++) {
          const double v = fma(-a[kk * LD], g, r[kk * LD]);
          g = fma(v, ib[kk * LD], v * lo[kk * LD]);
          r[kk * LD] = g;
        }
      }
    }
    __syncthreads();
  }
  if (warp == 2) bad = exp_field(g) == 0x7ff;  // an infinity or a NaN lasts to the end of its system
  if (bad) atomicOr(&again, 1u << (lane % S));
  // back substitution, last tile first: arrays 0 gamm, 1 cc/beta, 2 the solution
  double xn = 0.0;
  for (int i = 0; i < nt + 3; i++) {
    if (warp == 0) {
      if (i < nt) {
        const int t = nt - 1 - i;
        double *gm = tile(i, 0), *f = tile(i, 1);
#pragma unroll
        for (int e = lane; e < KT * S; e += 32) {
          const int kk = e % KT, s = e / KT, k = t * KT + kk, o = kk * LD + s;
          const size_t q = base + (size_t)s * n + k;
          if (s < ns && k < n) {
            cp_async8(gm + o, sol + q);
            cp_async8(f + o, gamm + q);
          } else {
            gm[o] = 0.0;
            f[o] = 0.0;
          }
        }
      }
      cp_async_commit();
      cp_async_wait<1>();
    } else if (warp == 1) {
      if (i >= 2 && i - 2 < nt && lane < S) {
        const double *gm = tile(i - 2, 0) + lane, *f = tile(i - 2, 1) + lane;
        double *o = tile(i - 2, 2) + lane;
#pragma unroll
        for (int kk = KT - 1; kk >= 0; kk--) {
          xn = fma(-f[kk * LD], xn, gm[kk * LD]);
          o[kk * LD] = xn;
        }
      }
    } else if (warp == 2) {
      if (i >= 3) {
        const int t = nt - 1 - (i - 3);
        const double *o = tile(i - 3, 2);
#pragma unroll
        for (int e = lane; e < KT * S; e += 32) {
          const int kk = e % KT, s = e / KT, k = t * KT + kk;
          if (s < ns && k < n) sol[base + (size_t)s * n + k] = o[kk * LD + s];
        }
      }
    }
    __syncthreads();
  }
  if (threadIdx.x < ns && (again >> threadIdx.x & 1)) {
    const size_t o = base + (size_t)threadIdx.x * n;
    thomas_plain(rhs + o, sol + o, aa + o, bb + o, cc + o, gamm + o, n);
  }
}

// S systems per CTA: 8 keeps a batch of up to 2 x 148 x 8 systems on CTAs of
// their own (the chain's length sets the time, so more systems per CTA gain
// nothing there); larger batches are bound by throughput and take 16.
static const void *thomas_kernel(int nbatch, int *s, size_t *smem) {
  *s = nbatch <= 2 * 148 * 8 ? 8 : 16;
  *smem = sizeof(double) * kThomRing * kThomArr * kThomKT * (*s + 1);
  return *s == 8 ? (const void *)k_thomas<8> : (const void *)k_thomas<16>;
}

// returns the error of this launch alone: one that an earlier, unrelated
// launch left pending on the thread is neither reported nor cleared
static cudaError_t launch_thomas(const double *rhs, double *sol, const double *aa, const double *bb, const double *cc,
                                 double *gamm, int n, int nbatch, cudaStream_t st) {
  int s;
  size_t smem;
  const void *kern = thomas_kernel(nbatch, &s, &smem);
  cudaError_t e = allow_dyn_smem(kern, smem);
  if (e) return e;
  void *args[] = {(void *)&rhs, (void *)&sol, (void *)&aa, (void *)&bb, (void *)&cc, (void *)&gamm,
                  (void *)&n, (void *)&nbatch};
  return cudaLaunchKernel(kern, dim3((nbatch + s - 1) / s), dim3(kThomThreads), args, smem, st);
}

cudaError_t launch_thomas_batched(const double *rhs, double *sol, const double *aa, const double *bb,
                                  const double *cc, int n, int nbatch, cudaStream_t s) {
  double *gamm = nullptr;
  cudaError_t e = cudaMallocAsync(&gamm, sizeof(double) * (size_t)n * nbatch, s);
  if (e) return e;
  e = launch_thomas(rhs, sol, aa, bb, cc, gamm, n, nbatch, s);
  cudaFreeAsync(gamm, s);
  return e;
}

// Block Thomas with identity off-diagonal blocks.  One CTA per system; the
// m x m blocks live in shared memory and are inverted with Doolittle LU
// exactly as btrithom.F90:99-177 (no pivoting); delta_k = beta_k^{-1} is kept
// in global scratch for the back substitution.
__device__ void blk_inverse(double *a, double *cinv, double *L, double *U, double *d, double *x, int n) {
  // a, L, U: n x n column-major in shared memory; serial per CTA thread 0..n-1
  int t = threadIdx.x;
  for (int i = t; i < n * n; i += blockDim.x) {
    L[i] = 0.0;
    U[i] = 0.0;
  }
  __syncthreads();
  for (int k = 0; k < n - 1; k++) {
    for (int i = k + 1 + t; i < n; i += blockDim.x) {
      double coeff = a[i + n * k] / a[k + n * k];
      L[i + n * k] = coeff;
      for (int j = k + 1; j < n; j++) a[i + n * j] = a[i + n * j] - coeff * a[k + n * j];
    }
    __syncthreads();
  }
  for (int i = t; i < n; i += blockDim.x) L[i + n * i] = 1.0;
  for (int j = t; j < n; j += blockDim.x)
    for (int i = 0; i <= j; i++) U[i + n * j] = a[i + n * j];
  __syncthreads();
  // columns of the inverse: thread k solves column k
  for (int k = t; k < n; k += blockDim.x) {
    double *dd = d + (size_t)k * n, *xx = x + (size_t)k * n;
    for (int i = 0; i < n; i++) {
      double v = (i == k) ? 1.0 : 0.0;
      for (int j = 0; j < i; j++) v = v - L[i + n * j] * dd[j];
      dd[i] = v;
    }
    xx[n - 1] = dd[n - 1] / U[(n - 1) + n * (n - 1)];
    for (int i = n - 2; i >= 0; i--) {
      double v = dd[i];
      for (int j = n - 1; j >= i + 1; j--) v = v - U[i + n * j] * xx[j];
      xx[i] = v / U[i + n * i];
    }
    for (int i = 0; i < n; i++) cinv[i + n * k] = xx[i];
  }
  __syncthreads();
}

__global__ void k_bthom(const double *__restrict__ rhs, double *__restrict__ sol, const double *__restrict__ b1,
                        const double *__restrict__ b2, const double *__restrict__ b3, int m, int n,
                        double *__restrict__ work) {
  extern __shared__ double sm[];
  const int sys = blockIdx.x;
  const size_t so = (size_t)sys * m * n;
  double *delta = work + (size_t)sys * ((size_t)m * m * n + (size_t)m * n + 2 * (size_t)m * m);
  double *gamm = delta + (size_t)m * m * n;
  double *dscr = gamm + (size_t)m * n;  // per-column forward vectors (m*m)
  double *xscr = dscr + (size_t)m * m;
  double *beta = sm, *L = sm + m * m, *U = sm + 2 * m * m, *tmp = sm + 3 * m * m;
  const int t = threadIdx.x;
  for (int k = 0; k < n; k++) {
    const double *B1 = b1 + so + (size_t)k * m, *B2 = b2 + so + (size_t)k * m, *B3 = b3 + so + (size_t)k * m;
    for (int i = t; i < m * m; i += blockDim.x) {
      int r = i % m, c = i / m;
      double v = 0.0;
      if (r == c) v = B2[r];
      if (r == c + 1) v = B1[r];
      if (c == r + 1) v = B3[r];
      if (k > 0) v = v - 1.0 * delta[(size_t)(k - 1) * m * m + i];
      beta[i] = v;
    }
    // gamm_k = rhs_k - delta_{k-1} gamm_{k-1}
    for (int i = t; i < m; i += blockDim.x) {
      double s = 0.0;
      if (k > 0)
        for (int j = 0; j < m; j++) s += delta[(size_t)(k - 1) * m * m + i + (size_t)m * j] * gamm[(size_t)(k - 1) * m + j];
      gamm[(size_t)k * m + i] = rhs[so + (size_t)k * m + i] - s;
    }
    __syncthreads();
    blk_inverse(beta, delta + (size_t)k * m * m, L, U, dscr, xscr, m);
    __syncthreads();
  }
  // sol_n = delta_n gamm_n ; sol_k = -delta_k (sol_{k+1} - gamm_k)
  for (int i = t; i < m; i += blockDim.x) {
    double s = 0.0;
    for (int j = 0; j < m; j++) s += delta[(size_t)(n - 1) * m * m + i + (size_t)m * j] * (-gamm[(size_t)(n - 1) * m + j]);
    sol[so + (size_t)(n - 1) * m + i] = -1.0 * s;
  }
  __syncthreads();
  for (int k = n - 2; k >= 0; k--) {
    for (int j = t; j < m; j += blockDim.x) tmp[j] = sol[so + (size_t)(k + 1) * m + j] - gamm[(size_t)k * m + j];
    __syncthreads();
    for (int i = t; i < m; i += blockDim.x) {
      double s = 0.0;
      for (int j = 0; j < m; j++) s += delta[(size_t)k * m * m + i + (size_t)m * j] * tmp[j];
      sol[so + (size_t)k * m + i] = -1.0 * s;
    }
    __syncthreads();
  }
}

cudaError_t launch_bthom_batched(const double *rhs, double *sol, const double *b1, const double *b2,
                                 const double *b3, int m, int n, int nbatch, double *work, cudaStream_t s) {
  size_t sm = sizeof(double) * (3 * (size_t)m * m + m);
  cudaError_t e = allow_dyn_smem(k_bthom, sm);
  if (e) return e;
  k_bthom<<<nbatch, 128, sm, s>>>(rhs, sol, b1, b2, b3, m, n, work);
  return cudaGetLastError();
}

}  // namespace vr

using namespace vr;

static int copy_in(const double *h, double **d, size_t n) {
  if (cudaMalloc(d, n * sizeof(double)) != cudaSuccess) return VR_ERR_OOM;
  if (cudaMemcpy(*d, h, n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess) return VR_ERR_CUDA;
  return VR_OK;
}

extern "C" int vr_solve_lap_thom(const double *rhs, double *sol, const double *aa, const double *bb,
                                 const double *cc, int32_t n, int32_t nbatch) {
  if (!rhs || !sol || !aa || !bb || !cc || n < 1 || nbatch < 1) return VR_ERR_ARG;
  size_t N = (size_t)n * nbatch;
  double *d[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  const double *h[4] = {rhs, aa, bb, cc};
  int rc = VR_OK;
  for (int i = 0; i < 4 && rc == VR_OK; i++) rc = copy_in(h[i], &d[i], N);
  if (rc == VR_OK && cudaMalloc(&d[4], N * sizeof(double)) != cudaSuccess) rc = VR_ERR_OOM;
  if (rc == VR_OK && launch_thomas_batched(d[0], d[4], d[1], d[2], d[3], n, nbatch, 0) != cudaSuccess) rc = VR_ERR_CUDA;
  if (rc == VR_OK && cudaMemcpy(sol, d[4], N * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) rc = VR_ERR_CUDA;
  for (double *p : d)
    if (p) cudaFree(p);
  return rc;
}

// ---------------------------------------------------------------------------
// vr_solve_lap_thom_noalloc: the batched Thomas solve on caller-owned device
// arrays, with its gamm scratch in a fixed array of this library instead of a
// per-call allocation.  It is meant for hosts that size all device memory once
// at start-up and then run a time loop that must not allocate: a per-call
// cudaMallocAsync can fail with out-of-memory halfway through a long run when
// other work has taken the pool, and it adds allocator work to every call.
// The scratch is one file-scope array per device, shared by every call on
// that device.  Every call writes the scratch rows it later reads, so nothing
// in it needs to start at zero; two calls that execute at the same time on
// one device (different streams or host threads) use the same rows and
// corrupt each other's results, so such calls must be ordered, e.g. on one
// stream.  The array's address is looked up once per device on the first call
// (cudaGetSymbolAddress), which may load the module; make that first call
// before any stream capture.  The address stays cached for the life of the
// process: after cudaDeviceReset (or anything else that destroys the device's
// primary context) the module may load at another address, and this entry
// point must not be called on that device again.
static __device__ __align__(256) double g_thom_scratch[VR_THOM_NOALLOC_MAX];

namespace {
constexpr int kMaxDevices = 64;
std::atomic<double *> g_thom_scratch_ptr[kMaxDevices];
}  // namespace

extern "C" int vr_solve_lap_thom_noalloc(const double *rhs, double *sol, const double *aa, const double *bb,
                                         const double *cc, int32_t n, int32_t nbatch, void *cuda_stream) {
  if (!rhs || !sol || !aa || !bb || !cc || n < 1 || nbatch < 1) return VR_ERR_ARG;
  if ((int64_t)n * nbatch > (int64_t)VR_THOM_NOALLOC_MAX) return VR_ERR_SCRATCH;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return VR_ERR_NODEVICE;
  if (dev >= kMaxDevices) return VR_ERR_ARG;
  double *gamm = g_thom_scratch_ptr[dev].load(std::memory_order_acquire);
  if (!gamm) {
    void *addr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&addr, g_thom_scratch);
    if (e != cudaSuccess || !addr) return VR_ERR_CUDA;
    gamm = static_cast<double *>(addr);
    g_thom_scratch_ptr[dev].store(gamm, std::memory_order_release);
  }
  return launch_thomas(rhs, sol, aa, bb, cc, gamm, n, nbatch, static_cast<cudaStream_t>(cuda_stream)) == cudaSuccess
             ? VR_OK
             : VR_ERR_CUDA;
}

extern "C" int vr_solve_lap_bthom(const double *rhs, double *sol, const double *b1, const double *b2,
                                  const double *b3, int32_t m, int32_t n, int32_t nbatch) {
  if (!rhs || !sol || !b1 || !b2 || !b3 || m < 1 || n < 1 || nbatch < 1 || m > 64) return VR_ERR_ARG;
  size_t N = (size_t)m * n * nbatch;
  double *d[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  const double *h[4] = {rhs, b1, b2, b3};
  int rc = VR_OK;
  for (int i = 0; i < 4 && rc == VR_OK; i++) rc = copy_in(h[i], &d[i], N);
  size_t wsz = (size_t)nbatch * ((size_t)m * m * n + (size_t)m * n + 2 * (size_t)m * m);
  if (rc == VR_OK && cudaMalloc(&d[4], N * sizeof(double)) != cudaSuccess) rc = VR_ERR_OOM;
  if (rc == VR_OK && cudaMalloc(&d[5], wsz * sizeof(double)) != cudaSuccess) rc = VR_ERR_OOM;
  if (rc == VR_OK && launch_bthom_batched(d[0], d[4], d[1], d[2], d[3], m, n, nbatch, d[5], 0) != cudaSuccess)
    rc = VR_ERR_CUDA;
  if (rc == VR_OK && cudaMemcpy(sol, d[4], N * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) rc = VR_ERR_CUDA;
  for (double *p : d)
    if (p) cudaFree(p);
  return rc;
}
