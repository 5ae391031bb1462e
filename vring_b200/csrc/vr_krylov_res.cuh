// vr_krylov_res.cuh -- CG on the axisymmetric operator with every vector
// resident on the chip (included by vr_krylov.cu).
//
// An iteration moves 40 MB through L2 when its kernels stream the vectors, yet
// all of them at 512 x 1024 are 20 MB, less than the registers of the chip.  So one cooperative kernel runs many iterations with
// the vectors in registers: a CTA owns nseg x C consecutive z planes, a thread
// one radial index j of C of them (nseg = 512 / nr segments side by side).
// Radial neighbours come from a shared-memory copy of the CTA's planes, z
// neighbours from the thread's own registers, from the next segment's planes
// in shared memory, or, at the CTA's ends, from the neighbouring CTA.
//
// What is left per iteration is the latency of its global sums.  A sum is one
// exchange: every CTA stores its partials into its own slot and reads the
// slots of all CTAs, adding them in the same order everywhere, so all CTAs
// compute the same scalars and no CTA waits for one that broadcasts.  A double
// travels as two 8-byte words, each half a value and half the exchange's
// number, so a reader knows a value from its stale predecessor by looking at
// it, and neither a fence nor a flag follows the data; the planes at a CTA's
// ends travel the same way beside the sums that need them anyway.  A CTA
// reuses a slot two exchanges later, when every CTA has contributed to the
// exchange in between and so has read it; an end plane is rewritten an
// iteration later for the same reason.
//
// Every wait is bounded (kWaitLimitNs): a CTA that gives up sets flags[3] and
// leaves, the others then run into their own limits, and the host reports
// VR_ERR_TIMEOUT.  The launch is cooperative, so all CTAs are resident.
//
// us per iteration of Jacobi CG, streaming kernels / resident: 20.2 / 6.3 at
// 512 x 1024, 12.1 / 4.6 at 128 x 256.  (BiCGSTAB the same way took 10.4 for
// 35.9, but its iterates depend on the order of the sums: two orders, both
// converged to 1e-12, answer 1e-9 apart, and it breaks down in one and not in
// the other, so it keeps the streaming kernels and their order.)  An exchange of one double per CTA between 148 CTAs takes 1.4 us
// beyond the sums inside the CTA (0.25): one 128-byte line per CTA, the slots
// packed side by side take 3.2 (the lines are then written by eight CTAs
// while all read them), one CTA that adds and broadcasts 1.9, a counter with
// fences 2.0, sums in groups of twelve 4.5.
#pragma once

#include "vr_tma.cuh"

namespace vr {

constexpr int kResThreads = 512;  // columns x segments of a CTA, at most
constexpr int kResMaxC = 8;       // planes per thread
constexpr int kResIters = 512;    // iterations per launch
constexpr int kResSlotWords = 16; // a 128-byte line per CTA, exchange and copy (up to four values)
constexpr int kResCopies = 4;     // of each slot, read by a quarter of the CTAs each
constexpr int kResMaxCtas = 256;  // a CTA's first 256 threads read one slot each

struct ResArg {
  int nr, nz, nseg;
  const double *aw, *ae, *az, *dinv;
  double gam;
  double *x, *r, *p;
  double *sc;
  int *flags;
  unsigned long long *slots;  // [2][kResCopies][CTAs][kResSlotWords]
  unsigned long long *ends;   // [CTAs][bottom, top][nr][2]
  unsigned epoch;             // number of the launch's first exchange
};

__device__ __forceinline__ void put_tagged(unsigned long long *a, double v, unsigned tag) {
  const unsigned long long t = (unsigned long long)tag << 32;
  const unsigned long long lo = t | (unsigned)__double2loint(v), hi = t | (unsigned)__double2hiint(v);
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(a), "l"(lo), "l"(hi) : "memory");
}
// Waits for exchange `tag`; try_get is one attempt.  False after the limit.
template <class F>
__device__ __forceinline__ bool wait_tagged(const F &try_get) {
  unsigned long long t0 = 0;
  for (unsigned n = 1; !try_get(); n++) {
    if ((n & 255) == 0) {  // the timer is read rarely
      const unsigned long long t = global_ns();
      if (t0 == 0)
        t0 = t;
      else if (t - t0 > kWaitLimitNs)
        return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool tagged(unsigned long long lo, unsigned long long hi, unsigned tag, double &v) {
  v = __hiloint2double((int)(unsigned)hi, (int)(unsigned)lo);
  return (unsigned)(lo >> 32) == tag && (unsigned)(hi >> 32) == tag;
}
__device__ __forceinline__ void ld_words(const unsigned long long *p, unsigned long long (&w)[2]) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w[0]), "=l"(w[1]) : "l"(p) : "memory");
}
__device__ __forceinline__ void ld_words(const unsigned long long *p, unsigned long long (&w)[4]) {
  asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
               : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
               : "l"(p)
               : "memory");
}
// the NV values of one slot, two per 32-byte load, all loads of an attempt in flight together
template <int NV>
__device__ __forceinline__ bool get_slot(const unsigned long long *p, unsigned tag, double (&v)[NV]) {
  return wait_tagged([&] {
    bool ok = true;
    if constexpr (NV == 1) {
      unsigned long long w[2];
      ld_words(p, w);
      ok = tagged(w[0], w[1], tag, v[0]);
    } else {
      unsigned long long w[(NV + 1) / 2][4];
#pragma unroll
      for (int i = 0; i < (NV + 1) / 2; i++) ld_words(p + 4 * i, w[i]);
#pragma unroll
      for (int i = 0; i < NV; i++) ok = tagged(w[i / 2][2 * (i & 1)], w[i / 2][2 * (i & 1) + 1], tag, v[i]) && ok;
    }
    return ok;
  });
}

__device__ __forceinline__ void give_up(const ResArg &a) {
  if (threadIdx.x == 0) atomicExch(a.flags + 3, 1);
}

struct ResShared {
  double part[kResThreads / 32][4];
  double tot[kResMaxCtas / 32][4];
};

// v[i] summed over all threads of all CTAs, the same bits in every thread;
// false (in every thread of the CTA) when a wait gave up
template <int NV>
__device__ __forceinline__ bool grid_sum(double (&v)[NV], const ResArg &a, unsigned tag, ResShared &sh) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < NV; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < NV; i++) sh.part[warp][i] = v[i];
  __syncthreads();
  unsigned long long *slots = a.slots + (size_t)(tag & 1) * kResCopies * gridDim.x * kResSlotWords;
  if (warp == 0) {
    double s[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) s[i] = lane < nw ? sh.part[lane][i] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < NV; i++) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
    if (lane < kResCopies)
#pragma unroll
      for (int i = 0; i < NV; i++)
        put_tagged(slots + ((size_t)lane * gridDim.x + blockIdx.x) * kResSlotWords + 2 * i, s[i], tag);
  }
  bool ok = true;
  const int nrw = ((int)gridDim.x + 31) >> 5;  // warps that read
  if (warp < nrw) {
    double got[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) got[i] = 0.0;
    if (threadIdx.x < gridDim.x)
      ok = get_slot(slots + ((size_t)(blockIdx.x % kResCopies) * gridDim.x + threadIdx.x) * kResSlotWords, tag, got);
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < NV; i++) got[i] += __shfl_xor_sync(0xffffffffu, got[i], o);
    if (lane == 0)
#pragma unroll
      for (int i = 0; i < NV; i++) sh.tot[warp][i] = got[i];
  }
  if (!__syncthreads_and(ok)) {
    give_up(a);
    return false;
  }
#pragma unroll
  for (int i = 0; i < NV; i++) {
    double s = 0.0;
    for (int w = 0; w < nrw; w++) s += sh.tot[w][i];
    v[i] = s;
  }
  return true;
}

// this thread's part of the operator
template <int C>
struct ResCell {
  int j, seg, k0, nc;  // radial index, segment, first plane, planes inside the grid (idle threads 0)
  bool wall, first, last;  // last radial row; segment at the CTA's lower, upper end
  double aw, ae, az;
  double *row;  // shared copy of (first plane, j)
  __device__ ResCell(const ResArg &a, double *planes) {
    const int t = threadIdx.x;
    seg = t / a.nr;
    j = t - seg * a.nr;
    const bool idle = seg >= a.nseg;
    if (idle) seg = 0;
    k0 = (blockIdx.x * a.nseg + seg) * C;
    nc = idle ? 0 : max(0, min(C, a.nz - k0));
    wall = j == a.nr - 1;
    first = !idle && seg == 0;
    last = !idle && seg == a.nseg - 1;
    aw = a.aw[j];
    ae = a.ae[j];
    az = a.az[j];
    row = planes + 1 + (size_t)seg * C * a.nr + j;
  }
  // copies this thread's planes into shared memory (the caller synchronises)
  __device__ void put(const ResArg &a, const double (&u)[C]) const {
#pragma unroll
    for (int c = 0; c < C; c++)
      if (c < nc) row[(size_t)c * a.nr] = u[c];
  }
  // y = S u; lo, hi: the planes beside the CTA, mean: of u's last radial row over z
  __device__ void apply(const ResArg &a, const double (&u)[C], double lo, double hi, double mean,
                        double (&y)[C]) const {
    if (!first && nc > 0) lo = row[-a.nr];
    if (!last && nc == C) hi = row[(size_t)C * a.nr];
#pragma unroll
    for (int c = 0; c < C; c++) {
      y[c] = 0.0;
      if (c >= nc) continue;
      const double *q = row + (size_t)c * a.nr;
      const double um = c > 0 ? u[c > 0 ? c - 1 : 0] : lo, up = c < C - 1 ? u[c < C - 1 ? c + 1 : 0] : hi;
      double s = aw * (u[c] - q[-1]);  // aw of the first row is 0
      if (wall)
        s += a.gam * mean;
      else
        s += ae * (u[c] - q[1]);
      if (k0 + c > 0) s += az * (u[c] - um);
      if (k0 + c < a.nz - 1) s += az * (u[c] - up);
      y[c] = s;
    }
  }
  // the CTA's end planes of u, and the neighbours'
  __device__ unsigned long long *end_slot(const ResArg &a, int cta, int top) const {
    return a.ends + 2 * (((size_t)cta * 2 + top) * a.nr + j);
  }
  __device__ void put_ends(const ResArg &a, const double (&u)[C], unsigned tag) const {
    if (first && blockIdx.x > 0) put_tagged(end_slot(a, blockIdx.x, 0), u[0], tag);
    if (last && blockIdx.x + 1 < gridDim.x) put_tagged(end_slot(a, blockIdx.x, 1), u[C - 1], tag);
  }
  // the neighbours' end planes; read after the sums of their exchange are in,
  // when they have as good as arrived: spinning on them meanwhile would put
  // every thread of the chip on L2 beside the sums
  __device__ bool get_ends(const ResArg &a, double &lo, double &hi, unsigned tag) const {
    const bool wlo = first && blockIdx.x > 0, whi = last && blockIdx.x + 1 < gridDim.x;
    if (!wlo && !whi) return true;
    const unsigned long long *pl = end_slot(a, wlo ? blockIdx.x - 1 : blockIdx.x + 1, wlo ? 1 : 0);
    const unsigned long long *ph = whi ? end_slot(a, blockIdx.x + 1, 0) : pl;
    double vl = 0.0, vh = 0.0;
    const bool ok = wait_tagged([&] {
      unsigned long long wl[2], wh[2];
      ld_words(pl, wl);
      ld_words(ph, wh);
      const bool okl = tagged(wl[0], wl[1], tag, vl), okh = tagged(wh[0], wh[1], tag, vh);
      return okl && okh;
    });
    if (wlo) lo = vl;
    if (whi) hi = vh;
    return ok;
  }
  // global index of plane c, and of the planes beside the CTA
  __device__ size_t at(const ResArg &a, int c) const { return j + (size_t)a.nr * (k0 + c); }
  __device__ void load(const ResArg &a, const double *g, double (&u)[C]) const {
#pragma unroll
    for (int c = 0; c < C; c++) u[c] = c < nc ? g[at(a, c)] : 0.0;
  }
  __device__ void store(const ResArg &a, double *g, const double (&u)[C]) const {
#pragma unroll
    for (int c = 0; c < C; c++)
      if (c < nc) g[at(a, c)] = u[c];
  }
  __device__ void load_ends(const ResArg &a, const double *g, double &lo, double &hi) const {
    lo = first && blockIdx.x > 0 ? g[j + (size_t)a.nr * (k0 - 1)] : 0.0;
    hi = last && blockIdx.x + 1 < gridDim.x ? g[j + (size_t)a.nr * (k0 + C)] : 0.0;
  }
};

// Up to kResIters CG iterations from the state (x, r, p, SC_BETA, SC_PMEAN,
// SC_RZ) that the setup or the previous launch left; the steps are those of
// k2d_cg_pq and k2d_cg_xr.  JAC: z = r / diag(S), else z = r.
// The argument stays in constant memory: a struct this small is otherwise held
// in registers over the loop, and the vectors spill (9.8 us per iteration at
// 512 x 1024 for 6.2).
template <int C, bool JAC>
__global__ void __launch_bounds__(kResThreads, 1) k2d_cg_res(const __grid_constant__ ResArg a) {
  extern __shared__ double planes[];
  __shared__ ResShared sh;
  if (a.flags[0]) return;
  const ResCell<C> e(a, planes);
  double x[C], r[C], p[C], q[C], di[C], dlo = 1.0, dhi = 1.0, plo, phi, zlo, zhi;
  e.load(a, a.x, x);
  e.load(a, a.r, r);
  e.load(a, a.p, p);
  e.load_ends(a, a.p, plo, phi);
  e.load_ends(a, a.r, zlo, zhi);
  if (JAC) {
    e.load(a, a.dinv, di);
    e.load_ends(a, a.dinv, dlo, dhi);
    zlo *= dlo;
    zhi *= dhi;
  }
  double be = a.sc[SC_BETA], pmean = a.sc[SC_PMEAN], rz = a.sc[SC_RZ], rr = 0.0, al = 0.0;
  const double stop = a.sc[SC_TOL2] * a.sc[SC_BB];
  int it = a.flags[1], done = 0;
  const int cap = a.flags[2];
  unsigned tag = a.epoch;
  bool ok = true;
  if (threadIdx.x == 0) planes[0] = planes[1 + (size_t)a.nseg * C * a.nr] = 0.0;
  for (int n = 0; n < kResIters && !done; n++) {
#pragma unroll
    for (int c = 0; c < C; c++) p[c] = (JAC ? r[c] * di[c] : r[c]) + be * p[c];
    plo = zlo + be * plo;
    phi = zhi + be * phi;
    e.put(a, p);
    if (!__syncthreads_and(ok)) return give_up(a);
    e.apply(a, p, plo, phi, pmean, q);
    double s1[1] = {0.0};
#pragma unroll
    for (int c = 0; c < C; c++) s1[0] += p[c] * q[c];
    if (!grid_sum(s1, a, tag++, sh)) return;
    al = rz / s1[0];
    double s2[4] = {0.0, 0.0, 0.0, 0.0}, z[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
      x[c] += al * p[c];
      r[c] -= al * q[c];
      z[c] = JAC ? r[c] * di[c] : r[c];
      s2[0] += r[c] * z[c];
      s2[1] += r[c] * r[c];
      if (e.wall) {
        s2[2] += z[c];
        s2[3] += p[c];
      }
    }
    e.put_ends(a, z, tag);
    if (!grid_sum(s2, a, tag, sh)) return;
    ok = e.get_ends(a, zlo, zhi, tag++);
    be = s2[0] / rz;
    rz = s2[0];
    rr = s2[1];
    pmean = (s2[2] + be * s2[3]) / a.nz;  // of the next direction
    it++;
    if (rr <= stop)
      done = 1;
    else if (it >= cap)
      done = 2;  // iteration cap: stop as not converged
  }
  e.store(a, a.x, x);
  e.store(a, a.r, r);
  e.store(a, a.p, p);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.sc[SC_ALPHA] = al;
    a.sc[SC_BETA] = be;
    a.sc[SC_PMEAN] = pmean;
    a.sc[SC_RZ] = rz;
    a.sc[SC_RR] = rr;
    a.flags[1] = it;
    a.flags[0] = done;
  }
}

// Planes per thread, segments and CTAs for a grid, or false: nr above 512
// (one thread per radial index), or more planes than C = 8 holds.  C is the
// smallest that fits one CTA per SM: 512 x 1024 spends 1.6 of its 6.1 us per
// iteration on seven planes per thread, while an exchange costs little more
// with 148 CTAs than with 64.
inline bool res_shape(int nr, int nz, int nsm, int *C, int *nseg, int *ctas) {
  if (nr > kResThreads) return false;
  nsm = nsm < kResMaxCtas ? nsm : kResMaxCtas;
  *nseg = kResThreads / nr;
  *C = (nz + *nseg * nsm - 1) / (*nseg * nsm);
  if (*C > kResMaxC) return false;
  *ctas = (nz + *nseg * *C - 1) / (*nseg * *C);
  return true;
}

}  // namespace vr
