// vr_unet.cu -- the learned preconditioner of the axisymmetric Krylov solve:
// a 4-level U-Net with BF16 weights and activations and FP32 accumulation,
// with its own forward, backward (data and weight gradients) and Adam kernels.
//
// Layout: activations are channels-last on the (nr_l x nz_l) grid of level l,
// pixel p = j + nr_l k (r fastest), element p * C + c.  A 3x3 layer's weights
// are [cout][tap][cin] with tap = 3 * dr + dz, dr, dz in {0, 1, 2} meaning the
// neighbour (j + dr - 1, k + dz - 1); zero padding at the grid edges.
//
// Network (no biases, identity activations, so the map is linear):
//   level 0..2 down: two 3x3 convs (cin -> c_l -> c_l), the second's output is
//   the skip tensor e_l; 2x2 average pooling to the next level;
//   level 3: two 3x3 convs (c_2 -> c_3 -> c_3);
//   level 2..0 up: nearest 2x upsampling of the level below, concatenated with
//   e_l (upsampled channels first), two 3x3 convs (-> c_l -> c_l);
//   head: 1x1 conv c_0 -> 1, FP32 output.
//
// The forward convolutions run on the tensor cores (k_conv3_tc) or, by flag, on
// the CUDA cores (k_conv3).  The gradients are FP32 throughout, on the CUDA
// cores: the data gradient is the convolution with the flipped weights
// (k_dgrad3), the weight gradient an outer product per pixel (k_wgrad3), added
// with FP32 atomics.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "vr_internal.cuh"
#include "vr_learned.cuh"
#include "vr_tma.cuh"
#include "vr_umma.cuh"

namespace vr {

constexpr int kUnetLayers = 15;  // 14 3x3 layers + the 1x1 head

struct UnetLayer {
  int cin, cout, level, taps;
  size_t woff;  // offset in the parameter vector
};

}  // namespace vr

struct vr_unet {
  std::atomic<int> refs{1};  // the caller, and every solver whose preconditioner it is
  int nr = 0, nz = 0, dev = 0, nsm = 148;
  int ch[4] = {};
  int pool = 2;  // pooling factor between levels
  std::string err;
  vr::UnetLayer L[vr::kUnetLayers];
  size_t nparam = 0;
  // parameters: FP32 master, BF16 copy, FP32 copy for the kernels, gradient,
  // Adam moments
  float *w32 = nullptr, *wk = nullptr, *gw = nullptr, *m1 = nullptr, *m2 = nullptr;
  __nv_bfloat16 *w16 = nullptr;
  __nv_bfloat16 *wpk = nullptr;  // per 3x3 layer [nout][9][cinp] BF16, zero padded (tensor-core form)
  size_t wpk_off[14] = {};
  bool cuda_cores = false;       // forward convolutions on CUDA cores instead of tensor cores
  unsigned *status = nullptr;    // bit 0: a bounded tensor-core wait gave up
  int64_t adam_t = 0;
  // activations (bf16) and their gradients (fp32), one per tensor slot
  __nv_bfloat16 *x0 = nullptr;            // input, 1 channel
  __nv_bfloat16 *a[20] = {};              // layer outputs, pooled and concatenated tensors
  float *g[20] = {};
  float *gx0 = nullptr;                   // input gradient (gradient check only)
  float *y = nullptr, *gy = nullptr;      // head output and its gradient
  double *xs = nullptr;                   // host-staging and training residual (double)
  double *dscal = nullptr;                // device scalars: loss accumulator, ss, e.r
  cudaStream_t stream = nullptr;
};

namespace vr {

__device__ __forceinline__ float tof(__nv_bfloat16 v) { return __bfloat162float(v); }

// two FP32 values in a 64-bit register pair; fma2 is one fused multiply-add
// (rounded to nearest) in each half.  Its rate is that of two scalar ones (an
// outer product in registers runs at 29 T multiply-adds per second either
// way); it leaves half of the issue slots to the loads and conversions.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
  return c;
}

// out[p][co] = sum_{tap, ci} in[p + off(tap)][ci] w[co][tap][ci]
template <int CO>
__global__ void __launch_bounds__(256) k_conv3(const __nv_bfloat16 *__restrict__ in, int H, int W, int cin,
                                             const float *__restrict__ w, int cout, __nv_bfloat16 *__restrict__ out) {
  extern __shared__ float sm[];
  float *tin = sm;                 // [18*18][17]
  float *tw = sm + 18 * 18 * 17;   // [CO][9][16]
  const int tj = threadIdx.x & 15, tk = threadIdx.x >> 4;
  const int j0 = blockIdx.x * 16, k0 = blockIdx.y * 16;
  float acc[CO];
#pragma unroll
  for (int c = 0; c < CO; c++) acc[c] = 0.f;
  for (int c0 = 0; c0 < cin; c0 += 16) {
    const int cc = min(16, cin - c0);
    for (int e = threadIdx.x; e < 18 * 18 * 16; e += 256) {
      const int ci = e & 15, pix = e >> 4;
      const int pj = pix % 18, pk = pix / 18;
      const int gj = j0 + pj - 1, gk = k0 + pk - 1;
      float v = 0.f;
      if (ci < cc && gj >= 0 && gj < H && gk >= 0 && gk < W) v = tof(in[((size_t)gj + (size_t)H * gk) * cin + c0 + ci]);
      tin[pix * 17 + ci] = v;
    }
    for (int e = threadIdx.x; e < CO * 9 * 16; e += 256) {
      const int ci = e & 15, t = (e >> 4) % 9, co = e / 144;
      float v = 0.f;
      if (co < cout && ci < cc) v = w[((size_t)co * 9 + t) * cin + c0 + ci];
      tw[e] = v;
    }
    __syncthreads();
#pragma unroll 1
    for (int t = 0; t < 9; t++) {
      const int dr = t / 3, dz = t % 3;
      const float *ip = tin + ((tj + dr) + 18 * (tk + dz)) * 17;
      float xin[16];
#pragma unroll
      for (int ci = 0; ci < 16; ci++) xin[ci] = ip[ci];
#pragma unroll
      for (int co = 0; co < CO; co++) {
        const float4 *wp = reinterpret_cast<const float4 *>(tw + (co * 9 + t) * 16);
        const float4 a = wp[0], b = wp[1], c = wp[2], d = wp[3];
        float s = acc[co];
        s = fmaf(xin[0], a.x, s);
        s = fmaf(xin[1], a.y, s);
        s = fmaf(xin[2], a.z, s);
        s = fmaf(xin[3], a.w, s);
        s = fmaf(xin[4], b.x, s);
        s = fmaf(xin[5], b.y, s);
        s = fmaf(xin[6], b.z, s);
        s = fmaf(xin[7], b.w, s);
        s = fmaf(xin[8], c.x, s);
        s = fmaf(xin[9], c.y, s);
        s = fmaf(xin[10], c.z, s);
        s = fmaf(xin[11], c.w, s);
        s = fmaf(xin[12], d.x, s);
        s = fmaf(xin[13], d.y, s);
        s = fmaf(xin[14], d.z, s);
        s = fmaf(xin[15], d.w, s);
        acc[co] = s;
      }
    }
    __syncthreads();
  }
  const int gj = j0 + tj, gk = k0 + tk;
  if (gj < H && gk < W) {
    __nv_bfloat16 *op = out + ((size_t)gj + (size_t)H * gk) * cout;
#pragma unroll
    for (int co = 0; co < CO; co++)
      if (co < cout) op[co] = __float2bfloat16_rn(acc[co]);
  }
}

// The same 3x3 convolution on the tensor cores (BF16 in, FP32 accumulate):
// an implicit GEMM over a patch of 8 (r) x 16 (z) output pixels per CTA,
// M = 128 pixels (row m = r + 8 z), N = NOUT output channels, K = 9 CINP
// (CINP, NOUT: cin and cout rounded up to 16).  The CTA copies its input halo
// (10 x 18 pixels x CINP channels, zero outside the grid) into shared memory
// once, as 16-byte chunks of 8 channels at ((hz CC + cc) 10 + hr) 16 bytes
// (CC = CINP / 8).  In that order the 8 pixels (hr .. hr + 7, hz) of one
// chunk column are 8 consecutive 16-byte rows: a K-major operand without
// swizzle (core matrices of 8 rows x 16 bytes, 160 bytes apart in K and
// CC 160 bytes apart in M).  So for tap (dr, dz) the A operand of the whole
// patch is the halo itself, read from the start chunk (dz CC + cc) 10 + dr:
// no im2col matrix is built.  The weights of the 9 taps are staged once in
// the same form (wpk [tap][cc][n][8]).  One thread issues the 9 x CINP / 16
// MMAs (M 128, N NOUT, K 16) and commits them to an mbarrier; the FP32
// accumulator stays in tensor memory (128 lanes = pixels, NOUT columns) until
// the epilogue, where each warp loads its 32 lanes and stores BF16.  The wait
// is bounded; one that gives up sets bit 0 of *status, and the CTA still
// waits (bounded) for its MMAs and frees its tensor memory.
//
// With skip set, the input is the decoder's concatenation, read where it
// lies instead of from a copy: channels [0, cin) are the coarse level `in`
// (H/F x W/F pixels, nearest upsampling by F) and channels
// [cin, cin + cskip) the skip tensor at full resolution.  Both channel counts
// are multiples of 8, so every 16-byte chunk comes from one of them.
constexpr int kConvTR = 8, kConvTZ = 16;  // pixel patch of a CTA (r x z)
constexpr int kConvHR = kConvTR + 2, kConvHZ = kConvTZ + 2;
#ifndef VR_CONV_CTAS
#define VR_CONV_CTAS 8
#endif
constexpr int kConvCtas = VR_CONV_CTAS;  // resident CTAs per SM, at most
// Grids of at most this many CTAs leave SMs free: their successor starts beside
// them and stages its weights meanwhile (pdl_trigger).  The coarse levels are
// chains of such kernels, 6 us each of which a third is staging: a learned
// solve at 512 x 1024 131 -> 117 ms, together with the other kernels' launches.
constexpr int kTriggerCtas = 148;

template <int CINP>
__host__ __device__ constexpr int conv_halo_bytes() {
  return kConvHR * kConvHZ * CINP * 2;
}
template <int CINP, int NOUT>
__host__ __device__ constexpr int conv_wstage_bytes() {
  return 9 * CINP * NOUT * 2;
}

// What follows a level's last convolution is taken in its epilogue (EPI), from
// the rounded values and in the order of the separate kernels, so with their
// bits:
//   kEpiHead: the 1 x 1 head y = sum_c out_c w_c (k_head); yl: a copy of the
//     last radial row (or null).  out may be null: only the training reads it.
//   kEpiPool: the F x F average pooling (k_pool), through the halo the products
//     have done with; a patch holds whole cells, since F divides 8.
// A learned solve at 512 x 1024 spares four launches and a 17 MB tensor written
// and read again per iteration: 0.225 -> 0.216 ms per iteration.
enum ConvEpiKind { kEpiNone = 0, kEpiHead, kEpiPool };
struct ConvEpi {
  const float *w;
  float *y, *yl;
  __nv_bfloat16 *pooled;
  int F;
};

// sum of the F x F pixels from src on (pitches dr, dz in 16-byte chunks), r
// fastest, times 1 / F^2
template <int F>
__device__ __forceinline__ uint4 pool_chunk(const uint4 *src, size_t dr, size_t dz) {
  float s[8];
#pragma unroll
  for (int i = 0; i < 8; i++) s[i] = 0.f;
#pragma unroll
  for (int z = 0; z < F; z++)
#pragma unroll
    for (int r = 0; r < F; r++) {
      const uint4 u = src[dz * z + dr * r];
      const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        s[2 * i] += __uint_as_float(w[i] << 16);
        s[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
      }
    }
  const float inv = 1.f / (float)(F * F);
  __align__(16) __nv_bfloat16 b[8];
#pragma unroll
  for (int i = 0; i < 8; i++) b[i] = __float2bfloat16_rn(inv * s[i]);
  return *reinterpret_cast<const uint4 *>(b);
}

template <int CINP, int NOUT, int EPI>
__global__ void __launch_bounds__(128) k_conv3_tc(const __nv_bfloat16 *in, int H, int W, int cin,
                                                const __nv_bfloat16 *skip, int cskip, int F,
                                                const __nv_bfloat16 *__restrict__ wpk, int cout,
                                                __nv_bfloat16 *__restrict__ out, unsigned *status, int npr,
                                                int npatch, ConvEpi epi) {
  static_assert(CINP % 16 == 0 && NOUT % 16 == 0 && NOUT <= 64, "tile shape");
  constexpr int CC = CINP / 8, HR = kConvHR, HZ = kConvHZ;
  constexpr uint32_t NCOLS = NOUT <= 32 ? 32 : 64;
  constexpr uint32_t IDESC = umma_idesc_bf16_f32(128, NOUT);
  extern __shared__ uint8_t smraw[];
  uint8_t *sm = (uint8_t *)(((uintptr_t)smraw + 127) & ~(uintptr_t)127);
  uint8_t *wst = sm;                                    // [tap][cc][n] 16-byte chunks
  uint8_t *halos = sm + conv_wstage_bytes<CINP, NOUT>();  // one or two of [hz][cc][hr] 16-byte chunks
  __shared__ uint64_t bar;
  __shared__ uint32_t tbase;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    tmem_alloc(&tbase, NCOLS);
    tmem_relinquish();
  }
  if (tid == 0) {
    mbar_init(&bar, 1);
    mbar_init_fence();
  }
  const int ctot = skip ? cin + cskip : cin;
  // the halo of a patch, pixels (j0 - 1 .. j0 + 8, k0 - 1 .. k0 + 16), a warp
  // per row of constant k: a lane keeps its pixel and chunk of the row
  // (consecutive lanes take consecutive chunks of a pixel, then the next pixel
  // in r), so a row costs it a pointer, a bounds test and the copy
  auto fetch = [&](int patch, uint8_t *halo) {
    const int j0 = (patch % npr) * kConvTR, k0 = (patch / npr) * kConvTZ;
    if (cin > 1) {
#pragma unroll
      for (int p0 = 0; p0 < HR * CC; p0 += 32) {
        const int p = p0 + lane, cc = p % CC, hr = p / CC, j = j0 + hr - 1, ci = cc * 8;
        const bool mine = p < HR * CC, jlive = mine && j >= 0 && j < H && ci < ctot;
        const bool full = !skip || ci >= cin;  // at this level's resolution
        const int sh = full ? 0 : F >> 1;      // F = 2, 4: shift by 1, 2
        const __nv_bfloat16 *src = full ? (skip ? skip + (size_t)j * cskip + (ci - cin) : in + (size_t)j * cin + ci)
                                        : in + (size_t)(j >> sh) * cin + ci;
        const size_t row = full ? (size_t)H * (skip ? cskip : cin) : (size_t)(H >> sh) * cin;
        uint8_t *dst = halo + (size_t)(cc * HR + hr) * 16;
        if (mine)
#pragma unroll
          for (int hz0 = 0; hz0 < HZ; hz0 += 4) {
            const int hz = hz0 + warp, k = k0 + hz - 1;
            const bool live = jlive && k >= 0 && k < W;
            if (hz < HZ)
              cp_async16(dst + (size_t)hz * (CC * HR * 16), live ? src + row * (k >> sh) : in, live ? 16u : 0u);
          }
      }
    } else {  // one channel: the first of a pixel's chunks, zeros beside it
      for (int e = tid; e < HR * HZ; e += 128) {
        const int hr = e % HR, hz = e / HR, j = j0 + hr - 1, k = k0 + hz - 1;
        const bool live = j >= 0 && j < H && k >= 0 && k < W;
        const unsigned v = live ? (unsigned)__bfloat16_as_ushort(in[(size_t)j + (size_t)H * k]) : 0u;
#pragma unroll
        for (int cc = 0; cc < CC; cc++)
          *reinterpret_cast<uint4 *>(halo + (size_t)((hz * CC + cc) * HR + hr) * 16) =
              make_uint4(cc == 0 ? v : 0u, 0u, 0u, 0u);
      }
    }
  };
  // the packed weights are already in the staged order
  for (int e = tid; e < 9 * CC * NOUT; e += 128) cp_async16(wst + (size_t)e * 16, wpk + (size_t)e * 8, 16u);
  pdl_wait();  // up to here: tensor memory and the weights
  if (gridDim.x <= kTriggerCtas) {
    // A CTA counts as soon as one of its threads triggers, and the successor's
    // CTAs, which wait for this grid to end, take tensor memory as they start:
    // all of an SM's while this CTA's warp 0 still asks for its own would
    // leave both waiting.  So not before every warp knows that it has it.
    __syncthreads();
    pdl_trigger();
  }
  int patch = blockIdx.x, buf = 0;
  uint32_t phase = 0;
  if (patch < npatch) fetch(patch, halos);
  cp_async_commit();
  for (; patch < npatch; phase ^= 1, buf ^= 1) {
    uint8_t *halo = halos + (size_t)buf * conv_halo_bytes<CINP>();
    cp_async_wait<0>();
    fence_proxy_async();  // the halo and weights, before the tensor cores read them
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tbase;
    if (tid == 0) {
#pragma unroll 1
      for (int t = 0; t < 9; t++) {
        const int dr = t / 3, dz = t % 3;  // tap t: neighbour (j + dr - 1, k + dz - 1)
#pragma unroll
        for (int ks = 0; ks < CINP / 16; ks++) {
          const uint64_t ad =
              umma_desc_plain(halo + (size_t)((dz * CC + 2 * ks) * HR + dr) * 16, HR * 16, CC * HR * 16);
          const uint64_t bd = umma_desc_plain(wst + (size_t)((t * CC + 2 * ks) * NOUT) * 16, NOUT * 16, 128);
          umma_bf16(tmem, ad, bd, IDESC, (t | ks) ? 1u : 0u);
        }
      }
      umma_commit(&bar);
    }
    __syncwarp();
    // the next patch's halo meanwhile (its buffer's products were waited for)
    const int next = patch + gridDim.x;
    if (next < npatch) fetch(next, halos + (size_t)(buf ^ 1) * conv_halo_bytes<CINP>());
    cp_async_commit();
    const bool ok = mbar_wait(&bar, phase);
    tc_fence_after();
    const int j0 = (patch % npr) * kConvTR, k0 = (patch / npr) * kConvTZ;
    const int mr = tid % kConvTR, mz = tid / kConvTR;  // this thread's row of D: pixel (j0 + mr, k0 + mz)
    const int j = j0 + mr, k = k0 + mz;
    const bool pin = j < H && k < W;
    const size_t p = (size_t)j + (size_t)H * k;
    float hs = 0.f;
#pragma unroll
    for (int c0 = 0; c0 < NOUT; c0 += 16) {
      float v[16];
      tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)c0, v);
      if (pin && ok && c0 < cout) {
        __nv_bfloat16 *dst = out + p * cout + c0;
        __align__(16) __nv_bfloat16 b[16];
#pragma unroll
        for (int i = 0; i < 16; i++) b[i] = __float2bfloat16_rn(v[i]);
        if (EPI != kEpiHead || out) {
          reinterpret_cast<uint4 *>(dst)[0] = reinterpret_cast<const uint4 *>(b)[0];
          if (c0 + 16 <= cout)  // channel counts are multiples of 8
            reinterpret_cast<uint4 *>(dst)[1] = reinterpret_cast<const uint4 *>(b)[1];
        }
        if constexpr (EPI == kEpiHead) {
#pragma unroll
          for (int i = 0; i < 16; i++)
            if (c0 + i < cout) hs = fmaf(__bfloat162float(b[i]), __ldg(epi.w + c0 + i), hs);
        }
        if constexpr (EPI == kEpiPool) {
          uint4 *px = reinterpret_cast<uint4 *>(halo) + (tid * cout + c0) / 8;
          px[0] = reinterpret_cast<const uint4 *>(b)[0];
          if (c0 + 16 <= cout) px[1] = reinterpret_cast<const uint4 *>(b)[1];
        }
      }
    }
    if constexpr (EPI == kEpiHead)
      if (pin && ok) {
        epi.y[p] = hs;
        if (epi.yl && j == H - 1) epi.yl[k] = hs;
      }
    if constexpr (EPI == kEpiPool) {
      static_assert(CINP == NOUT && conv_halo_bytes<CINP>() >= 128 * NOUT * 2, "the patch fits its halo");
      __syncthreads();
      const int F = epi.F, c8 = cout / 8, nj = kConvTR / F, nk = kConvTZ / F, H2 = H / F, W2 = W / F;
      for (int e = tid; e < nj * nk * c8; e += 128) {
        const int q = e % c8, J = e / c8 % nj, K = e / c8 / nj, gj = j0 / F + J, gk = k0 / F + K;
        if (gj >= H2 || gk >= W2) continue;
        const uint4 *src = reinterpret_cast<const uint4 *>(halo) + (size_t)(F * J + kConvTR * F * K) * c8 + q;
        reinterpret_cast<uint4 *>(epi.pooled)[((size_t)gj + (size_t)H2 * gk) * c8 + q] =
            F == 2 ? pool_chunk<2>(src, c8, kConvTR * c8) : pool_chunk<4>(src, c8, kConvTR * c8);
      }
    }
    tc_fence_before();
    // a wait that gave up ends the walk for the whole CTA
    if (!__syncthreads_and(ok)) {
      if (tid == 0) atomicOr(status, 1u);
      // the MMAs may still be reading shared memory and writing tensor memory
      (void)mbar_wait(&bar, phase);
      break;
    }
    patch = next;
  }
  cp_async_wait<0>();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, NCOLS);
}

// packed tensor-core weights in the order the convolution stages them:
// wpk[((tap CC + cc) nout + n) 8 + q] = bf16(w[n][tap][8 cc + q]) for n < cout,
// 8 cc + q < cin, zero elsewhere (CC = cinp / 8)
__global__ void k_wpack(const float *__restrict__ w, int cin, int cout, int cinp, int nout,
                        __nv_bfloat16 *__restrict__ wpk) {
  const int n_el = nout * 9 * cinp, cc_n = cinp / 8;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n_el; e += gridDim.x * blockDim.x) {
    const int q = e % 8, n = (e / 8) % nout, cc = (e / (8 * nout)) % cc_n, t = e / (8 * nout * cc_n);
    const int ci = 8 * cc + q;
    const float v = (n < cout && ci < cin) ? w[((size_t)n * 9 + t) * cin + ci] : 0.f;
    wpk[e] = __float2bfloat16_rn(v);
  }
}

// A 3x3 layer's input: channels [0, ca) from a and, when b is set, [ca, ca + cb)
// from b at full resolution with a one level down (nearest upsampling by F):
// the decoder's concatenation where it lies
struct ConvIn {
  const __nv_bfloat16 *a;
  int ca;
  const __nv_bfloat16 *b;
  int cb, F;
  __device__ __forceinline__ const __nv_bfloat16 *at(int j, int k, int H, int ci) const {
    if (!b) return a + ((size_t)j + (size_t)H * k) * ca + ci;
    if (ci < ca) return a + ((size_t)(j / F) + (size_t)(H / F) * (k / F)) * ca + ci;
    return b + ((size_t)j + (size_t)H * k) * cb + (ci - ca);
  }
};

// dw[co][tap][ci] += sum_p dout[p][co] in[p + off(tap)][ci]: an outer product
// per pixel, summed over the grid.  What bounds it is the FP32 pipe (6.1 G
// multiply-adds per sample at 512 x 1024), as long as the sums stay in
// registers and shared memory feeds them seldom: a thread holds 4 output x CIT
// input channels x 9 taps (CIT 4: 144 sums) and walks a line of pixels along
// r, so of the 3 x 3 input values only the three of the new column are loaded
// per pixel, with one load of the 4 gradients.  A CTA takes 16 output x 16
// input channels (CIT 1, the first layer: 16 x 1) of patches of R x NS
// pixels, one of its NS threads of equal channels per line, brought in by
// 16-byte asynchronous copies two patches ahead of each other (zero outside the
// grid).  It walks every gridDim.y-th patch and only then adds its threads'
// sums (shuffle, shared memory) and the result to dw by FP32 atomics.
// us at 512 x 1024 for 16 -> 16, 48 -> 16 and 1 -> 16 channels: 62, 185 and 23
// (19.5 T multiply-adds per second in the first two); one (output, input) pair
// per thread with ten scalar loads per nine multiply-adds, 4096 pixels per CTA:
// 830, 1350 and 830, and 410 to 950 on the coarser levels (now 8 to 49).
template <int CIT>
struct WgShape {
  static constexpr int OT = CIT == 4 ? 16 : 4;  // threads that share a line
  static constexpr int NS = 256 / OT;           // lines of a patch
  static constexpr int R = CIT == 4 ? 33 : 12;  // pixels of a line (a multiple of the window's 3 phases)
  static constexpr int IC = CIT == 4 ? 16 : 1;  // input channels of a CTA
  // floats between lines of the gradient tile: 16 beyond the line, so that two lines fill the banks
  static constexpr int DP = R * 16 + 16;
  static constexpr int IN_BYTES = CIT == 4 ? (NS + 2) * (R + 2) * 32 : (NS + 2) * (R + 3) * 4;
  static constexpr int STAGE = ((IN_BYTES + 15) & ~15) + NS * DP * 4;
};

template <int CIT>
__global__ void __launch_bounds__(256, 1) k_wgrad3(const float *__restrict__ dout, int H, int W, int cout, ConvIn in,
                                                 int cin, float *__restrict__ dw, int npr, int npatch) {
  using S = WgShape<CIT>;
  constexpr int NS = S::NS, R = S::R, DP = S::DP, NA = 4 * 9 * CIT;
  extern __shared__ uint8_t smraw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nci = (cin + S::IC - 1) / S::IC;
  const int ci0 = (blockIdx.x % nci) * S::IC, co0 = (blockIdx.x / nci) * 16;
  const int cig = CIT == 4 ? tid & 3 : 0, cog = CIT == 4 ? (tid >> 2) & 3 : tid & 3, line = tid / S::OT;
  auto stage_in = [&](int s) { return smraw + (size_t)s * S::STAGE; };
  auto stage_d = [&](int s) { return (float *)(smraw + (size_t)s * S::STAGE + ((S::IN_BYTES + 15) & ~15)); };
  auto fetch = [&](int patch, int s) {
    const int j0 = (patch % npr) * R, k0 = (patch / npr) * NS;
    if (CIT == 4) {
      uint8_t *si = stage_in(s);
      for (int e = tid; e < (NS + 2) * (R + 2) * 2; e += 256) {
        const int q = e & 1, pix = e >> 1, hr = pix % (R + 2), hz = pix / (R + 2);
        const int j = j0 + hr - 1, k = k0 + hz - 1, ci = ci0 + 8 * q;
        const bool live = j >= 0 && j < H && k >= 0 && k < W && ci < cin;
        cp_async16(si + (size_t)e * 16, live ? in.at(j, k, H, ci) : in.a, live ? 16u : 0u);
      }
    } else {  // one channel: plain loads, widened
      float *si = (float *)stage_in(s);
      for (int e = tid; e < (NS + 2) * (R + 2); e += 256) {
        const int hr = e % (R + 2), hz = e / (R + 2), j = j0 + hr - 1, k = k0 + hz - 1;
        const bool live = j >= 0 && j < H && k >= 0 && k < W;
        si[hz * (R + 3) + hr] = live ? tof(*in.at(j, k, H, 0)) : 0.f;
      }
    }
    float *sd = stage_d(s);
    for (int e = tid; e < NS * R * 4; e += 256) {
      const int q = e & 3, pix = e >> 2, hr = pix % R, hz = pix / R;
      const int j = j0 + hr, k = k0 + hz, co = co0 + 4 * q;
      const bool live = j < H && k < W && co < cout;
      cp_async16(sd + hz * DP + hr * 16 + 4 * q, live ? dout + ((size_t)j + (size_t)H * k) * cout + co : dout,
                 live ? 16u : 0u);
    }
    cp_async_commit();
  };
  // CIT 4: output channel a, input channels 2 c, 2 c + 1 (the widened input
  // comes in pairs, only the four gradients are copied into both halves);
  // CIT 1: output channels 2 a, 2 a + 1
  constexpr int PA = CIT == 4 ? 4 : 2, PC = CIT == 4 ? 2 : 1;
  f32x2 acc[PA][9][PC];
#pragma unroll
  for (int a = 0; a < PA; a++)
#pragma unroll
    for (int t = 0; t < 9; t++)
#pragma unroll
      for (int c = 0; c < PC; c++) acc[a][t][c] = 0ull;
  int s = 0, p = blockIdx.y;
  if (p < npatch) fetch(p, 0);
  for (; p < npatch; p += gridDim.y, s ^= 1) {
    const int nx = p + gridDim.y;
    if (nx < npatch) {
      fetch(nx, s ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const float *sd = stage_d(s) + line * DP + 4 * cog;
    // column hr (0 .. R + 1) of the halo rows line .. line + 2
    f32x2 w[3][3][PC];  // [column mod 3][dz]
    auto column = [&](int hr, f32x2 (&v)[3][PC]) {
#pragma unroll
      for (int dz = 0; dz < 3; dz++) {
        if constexpr (CIT == 4) {
          const uint2 u = *reinterpret_cast<const uint2 *>(stage_in(s) + ((size_t)(line + dz) * (R + 2) + hr) * 32 +
                                                           8 * cig);
          v[dz][0] = pack2(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u));
          v[dz][1] = pack2(__uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
        } else {
          const float f = ((const float *)stage_in(s))[(line + dz) * (R + 3) + hr];
          v[dz][0] = pack2(f, f);
        }
      }
    };
    column(0, w[0]);
    column(1, w[1]);
    const int rend = min(R, H - (p % npr) * R);  // pixels of the line inside the grid
#pragma unroll 1
    for (int r = 0; r < rend; r += 3) {
#pragma unroll
      for (int u = 0; u < 3; u++) {  // pixel r + u; past the line its gradient is 0
        column(r + u + 2, w[(u + 2) % 3]);
        f32x2 dd[PA];
        if constexpr (CIT == 4) {
          const float4 d = *reinterpret_cast<const float4 *>(sd + (r + u) * 16);
          dd[0] = pack2(d.x, d.x), dd[1] = pack2(d.y, d.y), dd[2] = pack2(d.z, d.z), dd[3] = pack2(d.w, d.w);
        } else {
          const ulonglong2 d = *reinterpret_cast<const ulonglong2 *>(sd + (r + u) * 16);
          dd[0] = d.x, dd[1] = d.y;
        }
#pragma unroll
        for (int dr = 0; dr < 3; dr++)
#pragma unroll
          for (int dz = 0; dz < 3; dz++)
#pragma unroll
            for (int a = 0; a < PA; a++)
#pragma unroll
              for (int c = 0; c < PC; c++)
                acc[a][3 * dr + dz][c] = fma2(dd[a], w[(u + dr) % 3][dz][c], acc[a][3 * dr + dz][c]);
      }
    }
    __syncthreads();  // the stage is refilled
  }
  // the lines' sums: lanes of a warp that differ in the line, then the warps
  float *red = (float *)smraw;  // [warp][sum][OT]
  constexpr int OT = S::OT;
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int t = 0; t < 9; t++)
#pragma unroll
      for (int c = 0; c < CIT; c++) {
        float v, v0, v1;
        unpack2(CIT == 4 ? acc[a][t][c / 2] : acc[a / 2][t][0], v0, v1);
        v = ((CIT == 4 ? c : a) & 1) ? v1 : v0;
#pragma unroll
        for (int o = 16; o >= OT; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane < OT) red[((size_t)warp * NA + (a * 9 + t) * CIT + c) * OT + lane] = v;
      }
  __syncthreads();
  for (int e = tid; e < NA * OT; e += 256) {
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q++) v += red[(size_t)q * NA * OT + e];
    const int l = e % OT, i = e / OT, c = i % CIT, t = (i / CIT) % 9, a = i / (CIT * 9);
    const int ci = ci0 + (CIT == 4 ? 4 * (l & 3) : 0) + c, co = co0 + 4 * (CIT == 4 ? l >> 2 : l) + a;
    if (ci < cin && co < cout) atomicAdd(dw + ((size_t)co * 9 + t) * cin + ci, v);
  }
}

// Data gradient: gin[p][ci] = sum_{tap, co} gout[p - off(tap)][co] w[co][tap][ci],
// the convolution with the flipped weights w[co][8 - tap], in FP32.  Bound by
// the FP32 pipe once the sums sit in registers: a thread holds PX pixels along
// r x 8 channels; per four output channels and row of taps it loads PX + 2
// pixels of 4 gradients, and per output channel 24 weights that its whole warp
// shares, for 24 PX multiply-adds (packed, two channels each).  A CTA takes
// tiles of 4 PX x 16 pixels x up to 48 channels (64 threads per 8 channels) in
// turn, 16 output channels at a time; gradients (channels-last as they lie,
// 4 floats after every PX pixels so that the strips of a quarter warp meet
// different banks) and weights of the next 16 arrive by asynchronous copies
// meanwhile.  PX = 2 where PX = 8 would leave SMs idle (the coarse levels).
// us at 512 x 1024 for 16 -> 16 and 16 -> 48 channels: 77 and 187; one pixel x
// all channels per thread: 139 and 373, and 47 to 180 on the coarser levels
// (now 15 to 57).
template <int PX>
struct DgShape {
  static constexpr int TR = 4 * PX, KC = 16;
  // floats of a halo row: pixels of KC, a gap of 4 after every PX, and 16
  // floats modulo 32 in all, so that two rows fill the banks
  static constexpr int RAW = (TR + 2) * KC + ((TR + 2) / PX) * 4;
  static constexpr int ROW = RAW + (48 - RAW % 32) % 32;
  static constexpr int GF = 18 * ROW;  // floats of a stage's gradients
};

template <int PX>
__global__ void __launch_bounds__(384) k_dgrad3(const float *__restrict__ gout, int H, int W, int cout,
                                              const float *__restrict__ w, int cin, float *__restrict__ gin, int ntr,
                                              int ntiles) {
  using S = DgShape<PX>;
  constexpr int KC = S::KC, TR = S::TR, ROW = S::ROW;
  extern __shared__ float smf[];
  const int tid = threadIdx.x, nth = blockDim.x, nch = nth / 8;
  const int strip = tid & 63, grp = tid >> 6, ci0 = blockIdx.y * nch;
  const int sr = (strip & 3) * PX, sz = strip >> 2;
  const int nk = (cout + KC - 1) / KC, stage_f = S::GF + KC * 9 * nch;
  auto goff = [](int hr) { return hr * KC + (hr / PX) * 4; };
  // stage s: the gradients of item (tile, 16 output channels) [18][ROW] and its weights [KC][dz][dr][nch]
  auto fetch = [&](int tile, int kch, int s) {
    float *sg = smf + (size_t)s * stage_f, *sw = sg + S::GF;
    const int j0 = (tile % ntr) * TR, k0 = (tile / ntr) * 16, c0 = kch * KC, kc = min(KC, cout - c0);
    for (int e = tid; e < 18 * (TR + 2) * (KC / 4); e += nth) {
      const int q = e & 3, pix = e >> 2, hr = pix % (TR + 2), hz = pix / (TR + 2);
      const int j = j0 + hr - 1, k = k0 + hz - 1;
      const bool live = 4 * q < kc && j >= 0 && j < H && k >= 0 && k < W;
      cp_async16(sg + hz * ROW + goff(hr) + 4 * q,
                 live ? gout + ((size_t)j + (size_t)H * k) * cout + c0 + 4 * q : gout, live ? 16u : 0u);
    }
    if (cin >= 8) {
      const int n4 = nch / 4;
      for (int e = tid; e < KC * 9 * n4; e += nth) {
        const int c = (e % n4) * 4, r = e / n4, t = r % 9, co = r / 9;  // t = 3 dz + dr
        const bool live = co < kc && ci0 + c < cin;
        cp_async16(sw + r * nch + c,
                   live ? w + ((size_t)(c0 + co) * 9 + 8 - 3 * (t % 3) - t / 3) * cin + ci0 + c : w, live ? 16u : 0u);
      }
    } else {  // one channel
      for (int e = tid; e < KC * 9 * nch; e += nth) {
        const int c = e % nch, r = e / nch, t = r % 9, co = r / 9;
        sw[e] = c < cin && co < kc ? w[((size_t)(c0 + co) * 9 + 8 - 3 * (t % 3) - t / 3) * cin + c] : 0.f;
      }
    }
    cp_async_commit();
  };
  f32x2 acc[PX][4];
  int s = 0, tile = blockIdx.x, kch = 0;
  if (tile < ntiles) fetch(tile, 0, 0);
  for (; tile < ntiles; s ^= 1) {
    int ntile = tile, nkch = kch + 1;
    if (nkch == nk) {
      nkch = 0;
      ntile += gridDim.x;
    }
    if (ntile < ntiles) {
      fetch(ntile, nkch, s ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    if (kch == 0) {
#pragma unroll
      for (int p = 0; p < PX; p++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[p][c] = 0ull;
    }
    const float *sg = smf + (size_t)s * stage_f, *sw = sg + S::GF;
    const int kq = min(KC, cout - kch * KC) / 4;
#pragma unroll 1
    for (int cq = 0; cq < kq; cq++) {
#pragma unroll 1
      for (int dz = 0; dz < 3; dz++) {
        const float *gp = sg + (sz + dz) * ROW + 4 * cq;
        float g[PX + 2][4];
#pragma unroll
        for (int i = 0; i < PX + 2; i++) {
          const float4 v = *reinterpret_cast<const float4 *>(gp + goff(sr) + i * KC + (i / PX) * 4);
          g[i][0] = v.x, g[i][1] = v.y, g[i][2] = v.z, g[i][3] = v.w;
        }
#pragma unroll
        for (int co = 0; co < 4; co++) {
          const float *wp = sw + ((4 * cq + co) * 9 + 3 * dz) * nch + 8 * grp;
          f32x2 g2[PX + 2];
#pragma unroll
          for (int i = 0; i < PX + 2; i++) g2[i] = pack2(g[i][co], g[i][co]);
#pragma unroll
          for (int dr = 0; dr < 3; dr++) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(wp + dr * nch);
            const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(wp + dr * nch + 4);
            const f32x2 wv[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
            for (int p = 0; p < PX; p++)
#pragma unroll
              for (int c = 0; c < 4; c++) acc[p][c] = fma2(g2[p + dr], wv[c], acc[p][c]);
          }
        }
      }
    }
    __syncthreads();  // the stage is refilled
    if (nkch == 0) {
      const int ci = ci0 + 8 * grp, j0 = (tile % ntr) * TR + sr, k = (tile / ntr) * 16 + sz;
      if (ci < cin && k < W) {
#pragma unroll
        for (int p = 0; p < PX; p++) {
          const int j = j0 + p;
          if (j >= H) continue;
          float *o = gin + ((size_t)j + (size_t)H * k) * cin + ci;
          if (cin >= 8) {  // a multiple of 8
            *reinterpret_cast<ulonglong2 *>(o) = make_ulonglong2(acc[p][0], acc[p][1]);
            *reinterpret_cast<ulonglong2 *>(o + 4) = make_ulonglong2(acc[p][2], acc[p][3]);
          } else {  // one channel
            float v, rest;
            unpack2(acc[p][0], v, rest);
            o[0] = v;
          }
        }
      }
    }
    tile = ntile;
    kch = nkch;
  }
}

// F x F average pooling (children summed in FP32, r fastest, then scaled by
// 1 / F^2) and its gradient; eight, then four channels per thread
template <int F>
__global__ void k_pool(const __nv_bfloat16 *in, int H, int W, int c, __nv_bfloat16 *__restrict__ out) {
  pdl_wait();
  if (gridDim.x <= kTriggerCtas) pdl_trigger();
  const int H2 = H / F, W2 = W / F, c8 = c / 8, n = H2 * W2 * c8;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int q = e % c8, p = e / c8, J = p % H2, K = p / H2;
    const uint4 *src = reinterpret_cast<const uint4 *>(in + ((size_t)F * J + (size_t)H * F * K) * c) + q;
    reinterpret_cast<uint4 *>(out)[e] = pool_chunk<F>(src, c8, (size_t)H * c8);
  }
}
// gin[p][c] += gout[parent(p)][c] / F^2
template <int F>
__global__ void k_pool_bwd(const float *__restrict__ gout, int H, int W, int c, float *__restrict__ gin) {
  const int H2 = H / F, c4 = c / 4, n = H * W * c4;
  const float inv = 1.f / (float)(F * F);
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int q = e % c4, p = e / c4, j = p % H, k = p / H;
    const float4 g = reinterpret_cast<const float4 *>(gout)[((size_t)(j / F) + (size_t)H2 * (k / F)) * c4 + q];
    float4 v = reinterpret_cast<float4 *>(gin)[e];
    v.x += inv * g.x;
    v.y += inv * g.y;
    v.z += inv * g.z;
    v.w += inv * g.w;
    reinterpret_cast<float4 *>(gin)[e] = v;
  }
}
// out[p] = [coarse[parent(p)] (ca channels), skip[p] (cb channels)]
__global__ void k_upcat(const __nv_bfloat16 *__restrict__ coarse, int ca, const __nv_bfloat16 *__restrict__ skip,
                        int cb, int H, int W, int F, __nv_bfloat16 *__restrict__ out) {
  const int c = ca + cb, H2 = H / F;
  const size_t n = (size_t)H * W * c;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const int ch = (int)(e % c);
    const size_t p = e / c;
    const int j = (int)(p % H), k = (int)(p / H);
    out[e] = ch < ca ? coarse[((size_t)(j / F) + (size_t)H2 * (k / F)) * ca + ch] : skip[p * cb + ch - ca];
  }
}
// gradient of k_upcat: gcoarse = sum over the F^2 children (r fastest), gskip =
// the skip part (its first contribution); a thread takes four channels of a
// coarse cell, and of its children's skip part
template <int F>
__global__ void k_upcat_bwd(const float *__restrict__ gout, int ca, int cb, int H, int W, float *__restrict__ gcoarse,
                            float *__restrict__ gskip) {
  const int H2 = H / F, W2 = W / F, c4 = (ca + cb) / 4, a4 = ca / 4, b4 = cb / 4, n = H2 * W2 * c4;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int q = e % c4, P = e / c4, J = P % H2, K = P / H2;
    const size_t p0 = (size_t)F * J + (size_t)H * F * K;
    const float4 *src = reinterpret_cast<const float4 *>(gout) + p0 * c4 + q;
    float4 v[F * F];
#pragma unroll
    for (int d = 0; d < F * F; d++) v[d] = src[((size_t)H * (d / F) + d % F) * c4];
    if (q < a4) {
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int d = 0; d < F * F; d++) {
        s.x += v[d].x;
        s.y += v[d].y;
        s.z += v[d].z;
        s.w += v[d].w;
      }
      reinterpret_cast<float4 *>(gcoarse)[(size_t)P * a4 + q] = s;
    } else {
#pragma unroll
      for (int d = 0; d < F * F; d++)
        reinterpret_cast<float4 *>(gskip)[(p0 + (size_t)H * (d / F) + d % F) * b4 + (q - a4)] = v[d];
    }
  }
}
// head: y[p] = sum_c in[p][c] w[c], eight channels per load; yl: a copy of the
// last radial row (or null)
__global__ void k_head(const __nv_bfloat16 *in, int P, int nr, int c, const float *__restrict__ w,
                       float *__restrict__ y, float *__restrict__ yl) {
  pdl_wait();
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
    float s = 0.f;
    for (int ch = 0; ch < c; ch += 8) {
      const uint4 u = *reinterpret_cast<const uint4 *>(in + (size_t)p * c + ch);
      const unsigned q[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        s = fmaf(__uint_as_float(q[i] << 16), w[ch + 2 * i], s);
        s = fmaf(__uint_as_float(q[i] & 0xffff0000u), w[ch + 2 * i + 1], s);
      }
    }
    y[p] = s;
    if (yl && p % nr == nr - 1) yl[p / nr] = s;
  }
}
// head gradient: gin[p][c] = gy[p] w[c]; gw[c] += sum_p gy[p] in[p][c]; a
// thread keeps four channels, so a warp writes whole pixels side by side
__global__ void __launch_bounds__(256) k_head_bwd(const __nv_bfloat16 *__restrict__ in, int P, int c,
                                                const float *__restrict__ w, const float *__restrict__ gy,
                                                float *__restrict__ gin, float *__restrict__ gw) {
  __shared__ float4 red[256];
  const int nq = c / 4, per = 256 / nq, q = threadIdx.x % nq, lp = threadIdx.x / nq;
  const float4 wq = *reinterpret_cast<const float4 *>(w + 4 * q);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (lp < per)
    for (int p = blockIdx.x * per + lp; p < P; p += gridDim.x * per) {
      const float g = gy[p];
      const uint2 u = *reinterpret_cast<const uint2 *>(in + (size_t)p * c + 4 * q);
      *reinterpret_cast<float4 *>(gin + (size_t)p * c + 4 * q) = make_float4(g * wq.x, g * wq.y, g * wq.z, g * wq.w);
      acc.x = fmaf(g, __uint_as_float(u.x << 16), acc.x);
      acc.y = fmaf(g, __uint_as_float(u.x & 0xffff0000u), acc.y);
      acc.z = fmaf(g, __uint_as_float(u.y << 16), acc.z);
      acc.w = fmaf(g, __uint_as_float(u.y & 0xffff0000u), acc.w);
    }
  red[threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.x < c) {
    float s = 0.f;
    for (int i = 0; i < per; i++) s += reinterpret_cast<const float *>(&red[i * nq + threadIdx.x / 4])[threadIdx.x % 4];
    atomicAdd(gw + threadIdx.x, s);
  }
}
// input: x[p] * D[p] / s -> bf16 (D = dscale or 1; s = sqrt(*ss / n) when ss is
// given, else 1 / inv_host)
__global__ void k_in(const double *x, int n, const double *ss, double inv_host, const double *dscale,
                     __nv_bfloat16 *__restrict__ xb, const int *flags) {
  pdl_wait();
  if (flags && flags[0]) return;
  const double inv = ss ? (*ss > 0 ? 1.0 / sqrt(*ss / n) : 0.0) : inv_host;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double v = x[i] * inv * (dscale ? dscale[i] : 1.0);
    xb[i] = __float2bfloat16_rn((float)v);
  }
}
// output: z = s y
__global__ void k_out(const float *__restrict__ y, int n, double s, double *__restrict__ z) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) z[i] = s * (double)y[i];
}
// weights: bf16 copy and the rounded FP32 copy used by the kernels
__global__ void k_wprep(const float *__restrict__ w32, size_t n, __nv_bfloat16 *__restrict__ w16,
                        float *__restrict__ wk) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const __nv_bfloat16 b = __float2bfloat16_rn(w32[i]);
    w16[i] = b;
    wk[i] = __bfloat162float(b);
  }
}
// Adam (Kingma & Ba 2015) on the FP32 master weights, gradient scaled by gs
// (no step on the gradient of a forward pass that gave up)
__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       size_t n, float lr, float gs, float b1, float b2, float c1, float c2, float eps,
                       const unsigned *status) {
  if (*status) return;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float gi = g[i] * gs;
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

static cudaError_t conv3(const __nv_bfloat16 *in, int H, int W, int cin, const float *w, int cout, __nv_bfloat16 *out,
                         cudaStream_t s) {
  const size_t smb = sizeof(float) * (18 * 18 * 17);
  dim3 g((H + 15) / 16, (W + 15) / 16);
  cudaError_t e;
#define VR_CONV_CASE(C)                                                                  \
  if (cout <= C) {                                                                       \
    const size_t sm = smb + sizeof(float) * C * 9 * 16;                                  \
    if ((e = allow_dyn_smem(k_conv3<C>, sm))) return e;                                  \
    k_conv3<C><<<g, 256, sm, s>>>(in, H, W, cin, w, cout, out);                          \
    return cudaGetLastError();                                                           \
  }
  VR_CONV_CASE(8)
  VR_CONV_CASE(16)
  VR_CONV_CASE(32)
  VR_CONV_CASE(48)
  VR_CONV_CASE(64)
#undef VR_CONV_CASE
  return cudaErrorInvalidValue;
}

template <int CINP, int NOUT>
static cudaError_t conv3_tc_n(const __nv_bfloat16 *in, int H, int W, int cin, const __nv_bfloat16 *skip, int cskip,
                              int F, const __nv_bfloat16 *wpk, int cout, __nv_bfloat16 *out, unsigned *status,
                              int nsm, cudaStream_t s, ConvEpi epi) {
  constexpr int halo = conv_halo_bytes<CINP>(), wst = conv_wstage_bytes<CINP, NOUT>();
  const int npr = (H + kConvTR - 1) / kConvTR, npatch = npr * ((W + kConvTZ - 1) / kConvTZ);
  // resident CTAs per SM with two halo buffers; one buffer where no CTA walks,
  // and a CTA per patch where two do not fit beside the weights (128 channels
  // to 64: 148 + 2 x 46 KB)
  constexpr int most = std::min(kConvCtas, 220 * 1024 / (128 + wst + 2 * halo + 1024));
  const int grid = most ? std::min(npatch, nsm * most) : npatch;
  const size_t sm = 128 + (size_t)wst + (size_t)(npatch > grid ? 2 : 1) * halo;
  auto kern = k_conv3_tc<CINP, NOUT, kEpiNone>;
  if (epi.w || epi.pooled) {  // as many channels in as out
    if constexpr (CINP == NOUT)
      kern = epi.w ? k_conv3_tc<CINP, NOUT, kEpiHead> : k_conv3_tc<CINP, NOUT, kEpiPool>;
    else
      return cudaErrorInvalidValue;
  }
  cudaError_t e = allow_dyn_smem(kern, sm);
  if (e) return e;
  return launch_pdl(kern, grid, 128, sm, s, in, H, W, cin, skip, cskip, F, wpk, cout, out, status, npr, npatch, epi);
}

template <int CINP>
static cudaError_t conv3_tc_c(const __nv_bfloat16 *in, int H, int W, int cin, const __nv_bfloat16 *skip, int cskip,
                              int F, const __nv_bfloat16 *wpk, int cout, __nv_bfloat16 *out, unsigned *status,
                              int nsm, cudaStream_t s, ConvEpi epi) {
  switch ((cout + 15) / 16) {
    case 1: return conv3_tc_n<CINP, 16>(in, H, W, cin, skip, cskip, F, wpk, cout, out, status, nsm, s, epi);
    case 2: return conv3_tc_n<CINP, 32>(in, H, W, cin, skip, cskip, F, wpk, cout, out, status, nsm, s, epi);
    case 3: return conv3_tc_n<CINP, 48>(in, H, W, cin, skip, cskip, F, wpk, cout, out, status, nsm, s, epi);
    case 4: return conv3_tc_n<CINP, 64>(in, H, W, cin, skip, cskip, F, wpk, cout, out, status, nsm, s, epi);
    default: return cudaErrorInvalidValue;
  }
}

// tensor-core 3x3 convolution: cin (+ cskip) up to 128, cout up to 64; with
// skip, the input is the concatenation of `in` upsampled by F and `skip`
static cudaError_t conv3_tc(const __nv_bfloat16 *in, int H, int W, int cin, const __nv_bfloat16 *wpk, int cout,
                            __nv_bfloat16 *out, unsigned *status, int nsm, cudaStream_t s,
                            const __nv_bfloat16 *skip = nullptr, int cskip = 0, int F = 1, ConvEpi epi = {}) {
  if (skip && ((cin & 7) || (cskip & 7))) return cudaErrorInvalidValue;
  const int ctot = cin + (skip ? cskip : 0);
  switch ((ctot + 15) / 16) {
#define VR_CONV_TC(CP) return conv3_tc_c<CP>(in, H, W, cin, skip, cskip, F, wpk, cout, out, status, nsm, s, epi)
    case 1: VR_CONV_TC(16);
    case 2: VR_CONV_TC(32);
    case 3: VR_CONV_TC(48);
    case 4: VR_CONV_TC(64);
    case 5: VR_CONV_TC(80);
    case 6: VR_CONV_TC(96);
    case 7: VR_CONV_TC(112);
    case 8: VR_CONV_TC(128);
#undef VR_CONV_TC
    default: return cudaErrorInvalidValue;
  }
}

static int round16(int x) { return (x + 15) / 16 * 16; }

// One CTA per SM: as many patch walkers per channel tile as fill the chip
template <int CIT>
static cudaError_t wgrad3_n(const float *dout, int H, int W, int cout, const ConvIn &in, int cin, float *dw, int nsm,
                            cudaStream_t s) {
  using S = WgShape<CIT>;
  const int npr = (H + S::R - 1) / S::R, npatch = npr * ((W + S::NS - 1) / S::NS);
  const int nt = ((cin + S::IC - 1) / S::IC) * ((cout + 15) / 16);
  const size_t sm = std::max((size_t)2 * S::STAGE, (size_t)8 * 4 * 9 * CIT * S::OT * sizeof(float));
  cudaError_t e = allow_dyn_smem(k_wgrad3<CIT>, sm);
  if (e) return e;
  k_wgrad3<CIT><<<dim3(nt, std::min(npatch, std::max(1, nsm / nt))), 256, sm, s>>>(dout, H, W, cout, in, cin, dw, npr,
                                                                                  npatch);
  return cudaGetLastError();
}
static cudaError_t wgrad3(const float *dout, int H, int W, int cout, const ConvIn &in, int cin, float *dw, int nsm,
                          cudaStream_t s) {
  return cin == 1 ? wgrad3_n<1>(dout, H, W, cout, in, cin, dw, nsm, s)
                  : wgrad3_n<4>(dout, H, W, cout, in, cin, dw, nsm, s);
}

template <int PX>
static cudaError_t dgrad3_n(const float *gout, int H, int W, int cout, const float *w, int cin, float *gin, int grp,
                            int ny, int nsm, cudaStream_t s) {
  using S = DgShape<PX>;
  const int ntr = (H + S::TR - 1) / S::TR, ntiles = ntr * ((W + 15) / 16);
  const size_t sm = 2 * sizeof(float) * (S::GF + (size_t)S::KC * 9 * 8 * grp);
  cudaError_t e = allow_dyn_smem(k_dgrad3<PX>, sm);
  if (e) return e;
  // resident CTAs per SM by shared memory; each then takes its share of the tiles
  const int per = std::max(1, (int)((size_t)(220 * 1024) / sm));
  k_dgrad3<PX><<<dim3(std::min(ntiles, std::max(1, nsm * per / ny)), ny), 64 * grp, sm, s>>>(gout, H, W, cout, w, cin,
                                                                                            gin, ntr, ntiles);
  return cudaGetLastError();
}
static cudaError_t dgrad3(const float *gout, int H, int W, int cout, const float *w, int cin, float *gin, int nsm,
                          cudaStream_t s) {
  const int groups = (cin + 7) / 8;  // of 8 channels
  const int tiles8 = ((H + 31) / 32) * ((W + 15) / 16);
  int grp = std::min(groups, 6), ny = (groups + grp - 1) / grp;
  if (tiles8 * ny >= nsm) return dgrad3_n<8>(gout, H, W, cout, w, cin, gin, (groups + ny - 1) / ny, ny, nsm, s);
  grp = std::min(groups, 2);
  ny = (groups + grp - 1) / grp;
  return dgrad3_n<2>(gout, H, W, cout, w, cin, gin, grp, ny, nsm, s);
}

static int grid_for(size_t n) { return (int)std::min<size_t>((n + 255) / 256, 148 * 8); }


// BF16 copy, rounded FP32 copy and the packed tensor-core weights of every
// 3x3 layer, from the FP32 master weights
static cudaError_t unet_prep_weights(vr_unet *u, cudaStream_t s) {
  k_wprep<<<grid_for(u->nparam), 256, 0, s>>>(u->w32, u->nparam, u->w16, u->wk);
  for (int i = 0; i < 14; i++) {
    const UnetLayer &L = u->L[i];
    const int cinp = round16(L.cin), nout = round16(L.cout);
    k_wpack<<<grid_for((size_t)nout * 9 * cinp), 256, 0, s>>>(u->wk + L.woff, L.cin, L.cout, cinp, nout,
                                                             u->wpk + u->wpk_off[i]);
  }
  return cudaGetLastError();
}

}  // namespace vr

using namespace vr;

static int unet_err(vr_unet *u, int code, const std::string &m) {
  if (u) u->err = m;
  return code;
}
#define U_CUDA(u, call)                                                                        \
  do {                                                                                         \
    cudaError_t e_ = (call);                                                                   \
    if (e_ != cudaSuccess) return unet_err((u), VR_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

namespace {
// activation slots: id, level, channels (filled at create)
enum Slot {
  S_E0A, S_E0, S_P1, S_E1A, S_E1, S_P2, S_E2A, S_E2, S_P3, S_B3A, S_B3,
  S_U2, S_D2A, S_D2, S_U1, S_D1A, S_D1, S_U0, S_D0A, S_D0, S_NSLOT
};
}  // namespace

struct UnetShapes {
  int lev[S_NSLOT], ch[S_NSLOT];
};

static UnetShapes shapes_of(const vr_unet *u) {
  UnetShapes s;
  const int *c = u->ch;
  const int L[S_NSLOT] = {0, 0, 1, 1, 1, 2, 2, 2, 3, 3, 3, 2, 2, 2, 1, 1, 1, 0, 0, 0};
  const int C[S_NSLOT] = {c[0], c[0], c[0], c[1], c[1], c[1], c[2], c[2], c[2], c[3], c[3],
                          c[3] + c[2], c[2], c[2], c[2] + c[1], c[1], c[1], c[1] + c[0], c[0], c[0]};
  for (int i = 0; i < S_NSLOT; i++) {
    s.lev[i] = L[i];
    s.ch[i] = C[i];
  }
  return s;
}

// the 14 3x3 layers: (input slot or -1 for x0, output slot)
static const int kConvIn[14] = {-1, S_E0A, S_P1, S_E1A, S_P2, S_E2A, S_P3, S_B3A, S_U2, S_D2A, S_U1, S_D1A, S_U0, S_D0A};
static const int kConvOut[14] = {S_E0A, S_E0, S_E1A, S_E1, S_E2A, S_E2, S_B3A, S_B3, S_D2A, S_D2, S_D1A, S_D1, S_D0A, S_D0};

static_assert(S_NSLOT <= 20, "tensor slots");

extern "C" int vr_unet_destroy(vr_unet *u);

extern "C" int vr_unet_create(const vr_unet_desc *d, uint64_t seed, vr_unet **out) {
  if (!d || !out) return VR_ERR_ARG;
  *out = nullptr;
  if (d->abi_version != VR_ABI_VERSION) return VR_ERR_DESC;
  const int F = d->pool == 0 ? 2 : d->pool;
  if (F != 2 && F != 4) return VR_ERR_DESC;
  const int F3 = F * F * F;
  if (d->nr < F3 || d->nz < F3 || d->nr % F3 || d->nz % F3 || (int64_t)d->nr * d->nz > ((int64_t)1 << 24))
    return VR_ERR_DESC;
  for (int l = 0; l < 4; l++)
    if (d->ch[l] < 8 || d->ch[l] > 64 || d->ch[l] % 8) return VR_ERR_DESC;  // a 3x3 layer's output <= 64
  if (d->ch[0] > 64) return VR_ERR_DESC;  // the head's gradient keeps c0 sums per thread
  if (d->ch[3] + d->ch[2] > 128 || d->ch[2] + d->ch[1] > 128 || d->ch[1] + d->ch[0] > 128) return VR_ERR_DESC;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0 || d->device < 0 || d->device >= ndev)
    return VR_ERR_NODEVICE;
  vr_unet *u = new (std::nothrow) vr_unet();
  if (!u) return VR_ERR_OOM;
  auto fail = [&](int code) {
    vr_unet_destroy(u);
    return code;
  };
  u->nr = d->nr;
  u->nz = d->nz;
  u->pool = F;
  u->dev = d->device;
  for (int l = 0; l < 4; l++) u->ch[l] = d->ch[l];
  if (cudaSetDevice(u->dev) != cudaSuccess) return fail(VR_ERR_CUDA);
  if (cudaDeviceGetAttribute(&u->nsm, cudaDevAttrMultiProcessorCount, u->dev) != cudaSuccess) return fail(VR_ERR_CUDA);
  if (cudaStreamCreateWithFlags(&u->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(VR_ERR_CUDA);
  const UnetShapes sh = shapes_of(u);
  size_t off = 0;
  for (int i = 0; i < 14; i++) {
    const int cin = kConvIn[i] < 0 ? 1 : sh.ch[kConvIn[i]];
    const int cout = sh.ch[kConvOut[i]];
    u->L[i] = UnetLayer{cin, cout, sh.lev[kConvOut[i]], 9, off};
    off += (size_t)cin * cout * 9;
  }
  u->L[14] = UnetLayer{u->ch[0], 1, 0, 1, off};
  off += u->ch[0];
  u->nparam = off;
  // He-style initialisation scaled for a linear network: each 3x3 layer
  // preserves the variance of its input (std = 1 / sqrt(9 cin)), from a
  // splitmix64 stream (Box-Muller)
  std::vector<float> w(u->nparam);
  uint64_t st = seed;
  auto next = [&]() {
    uint64_t z = (st += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  };
  auto unif = [&]() { return ((next() >> 11) + 0.5) * (1.0 / 9007199254740992.0); };
  const double pi = std::acos(-1.0);
  for (int i = 0; i < kUnetLayers; i++) {
    const double sd = 1.0 / std::sqrt((double)u->L[i].cin * u->L[i].taps);
    const size_t n = (size_t)u->L[i].cin * u->L[i].cout * u->L[i].taps;
    for (size_t e = 0; e < n; e++)
      w[u->L[i].woff + e] = (float)(sd * std::sqrt(-2.0 * std::log(unif())) * std::cos(2.0 * pi * unif()));
  }
  const size_t P0 = (size_t)u->nr * u->nz;
  float **fp[] = {&u->w32, &u->wk, &u->gw, &u->m1, &u->m2};
  for (float **p : fp)
    if (cudaMalloc(p, sizeof(float) * u->nparam) != cudaSuccess) return fail(VR_ERR_OOM);
  if (cudaMalloc(&u->w16, sizeof(__nv_bfloat16) * u->nparam) != cudaSuccess) return fail(VR_ERR_OOM);
  size_t npk = 0;
  for (int i = 0; i < 14; i++) {
    u->wpk_off[i] = npk;
    npk += (size_t)round16(u->L[i].cout) * 9 * round16(u->L[i].cin);
  }
  if (cudaMalloc(&u->wpk, sizeof(__nv_bfloat16) * npk) != cudaSuccess) return fail(VR_ERR_OOM);
  if (cudaMalloc(&u->status, sizeof(unsigned)) != cudaSuccess) return fail(VR_ERR_OOM);
  if (cudaMemsetAsync(u->status, 0, sizeof(unsigned), u->stream) != cudaSuccess) return fail(VR_ERR_CUDA);
  u->cuda_cores = (d->flags & VR_UNET_CUDA_CORES) != 0;
  if (cudaMalloc(&u->x0, sizeof(__nv_bfloat16) * P0) != cudaSuccess) return fail(VR_ERR_OOM);
  if (cudaMalloc(&u->y, sizeof(float) * P0) != cudaSuccess) return fail(VR_ERR_OOM);
  if (cudaMalloc(&u->gy, sizeof(float) * P0) != cudaSuccess) return fail(VR_ERR_OOM);
  if (cudaMalloc(&u->xs, sizeof(double) * P0) != cudaSuccess) return fail(VR_ERR_OOM);
  if (cudaMalloc(&u->dscal, sizeof(double) * 8) != cudaSuccess) return fail(VR_ERR_OOM);
  vr_unet *x = u;
  for (int i = 0; i < S_NSLOT; i++) {
    size_t div = 1;
    for (int l = 0; l < sh.lev[i]; l++) div *= (size_t)u->pool * u->pool;
    const size_t n = (P0 / div) * sh.ch[i];
    const bool cat = i == S_U2 || i == S_U1 || i == S_U0;  // copied by the CUDA-core form only
    if ((!cat || u->cuda_cores) && cudaMalloc(&x->a[i], sizeof(__nv_bfloat16) * n) != cudaSuccess)
      return fail(VR_ERR_OOM);
    if (cudaMalloc(&x->g[i], sizeof(float) * n) != cudaSuccess) return fail(VR_ERR_OOM);
  }
  if (cudaMalloc(&x->gx0, sizeof(float) * P0) != cudaSuccess) return fail(VR_ERR_OOM);
  // on the stream that goes on to use them: cudaMemcpy from pageable memory and
  // cudaMemset may return before the device has the bytes, in the order of the
  // legacy stream, which this one does not wait for
  if (cudaMemcpyAsync(u->w32, w.data(), sizeof(float) * u->nparam, cudaMemcpyHostToDevice, u->stream) != cudaSuccess ||
      cudaMemsetAsync(u->m1, 0, sizeof(float) * u->nparam, u->stream) != cudaSuccess ||
      cudaMemsetAsync(u->m2, 0, sizeof(float) * u->nparam, u->stream) != cudaSuccess)
    return fail(VR_ERR_CUDA);
  if (unet_prep_weights(u, u->stream) != cudaSuccess) return fail(VR_ERR_CUDA);
  if (cudaStreamSynchronize(u->stream) != cudaSuccess) return fail(VR_ERR_CUDA);
  *out = u;
  return VR_OK;
}

static void unet_free(vr_unet *u) {
  cudaSetDevice(u->dev);
  if (u->stream) cudaStreamSynchronize(u->stream);
  for (int i = 0; i < S_NSLOT; i++) {
    if (u->a[i]) cudaFree(u->a[i]);
    if (u->g[i]) cudaFree(u->g[i]);
  }
  if (u->gx0) cudaFree(u->gx0);
  float *fp[] = {u->w32, u->wk, u->gw, u->m1, u->m2, u->y, u->gy};
  for (float *p : fp)
    if (p) cudaFree(p);
  if (u->w16) cudaFree(u->w16);
  if (u->wpk) cudaFree(u->wpk);
  if (u->status) cudaFree(u->status);
  if (u->x0) cudaFree(u->x0);
  if (u->xs) cudaFree(u->xs);
  if (u->dscal) cudaFree(u->dscal);
  if (u->stream) cudaStreamDestroy(u->stream);
  delete u;
}

namespace vr {

void unet_hold(const vr_unet *u) { const_cast<vr_unet *>(u)->refs.fetch_add(1, std::memory_order_relaxed); }
void unet_drop(const vr_unet *u) {
  vr_unet *x = const_cast<vr_unet *>(u);
  if (x->refs.fetch_sub(1, std::memory_order_acq_rel) == 1) unet_free(x);
}

}  // namespace vr

extern "C" int vr_unet_destroy(vr_unet *u) {
  if (u) unet_drop(u);
  return VR_OK;
}

extern "C" const char *vr_unet_last_error(const vr_unet *u) { return u ? u->err.c_str() : "null network"; }

extern "C" int vr_unet_nparams(const vr_unet *u, int64_t *n) {
  if (!u || !n) return VR_ERR_ARG;
  *n = (int64_t)u->nparam;
  return VR_OK;
}

extern "C" int vr_unet_get_params(const vr_unet *u, float *w) {
  if (!u || !w) return VR_ERR_ARG;
  if (cudaSetDevice(u->dev) != cudaSuccess) return VR_ERR_CUDA;
  if (cudaMemcpy(w, u->w32, sizeof(float) * u->nparam, cudaMemcpyDeviceToHost) != cudaSuccess) return VR_ERR_CUDA;
  return VR_OK;
}

extern "C" int vr_unet_set_params(vr_unet *u, const float *w) {
  if (!u || !w) return VR_ERR_ARG;
  U_CUDA(u, cudaSetDevice(u->dev));
  U_CUDA(u, cudaMemcpyAsync(u->w32, w, sizeof(float) * u->nparam, cudaMemcpyHostToDevice, u->stream));
  U_CUDA(u, unet_prep_weights(u, u->stream));
  U_CUDA(u, cudaStreamSynchronize(u->stream));
  return VR_OK;
}

namespace vr {

// forward from u->x0 (bf16 input) to u->y (fp32); the tensor-core
// convolutions (and the weight gradients) read the decoder's concatenations
// where they lie, only the CUDA-core form copies them
static cudaError_t unet_fwd(const vr_unet *u, cudaStream_t s, float *yl = nullptr, bool keep = true) {
  const UnetShapes sh = shapes_of(u);
  const vr_unet *x = u;
  cudaError_t e;
  auto HW = [&](int lev, int &H, int &W) {
    H = u->nr;
    W = u->nz;
    for (int l = 0; l < lev; l++) H /= u->pool, W /= u->pool;
  };
  int H, W;
  const bool fuse = !u->cuda_cores;
  auto conv = [&](int li, int pooled = -1) -> cudaError_t {
    const UnetLayer &L = u->L[li];
    HW(L.level, H, W);
    const __nv_bfloat16 *in = kConvIn[li] < 0 ? u->x0 : x->a[kConvIn[li]];
    if (u->cuda_cores)
      return conv3(in, H, W, L.cin, u->wk + L.woff, L.cout, x->a[kConvOut[li]], s);
    return conv3_tc(in, H, W, L.cin, u->wpk + u->wpk_off[li], L.cout, x->a[kConvOut[li]], u->status, u->nsm, s,
                    nullptr, 0, 1, ConvEpi{nullptr, nullptr, nullptr, pooled < 0 ? nullptr : x->a[pooled], u->pool});
  };
  // the first convolution of a decoder level, on concat(upsample(coarse), skip)
  auto conv_cat = [&](int li, int coarse, int skip) -> cudaError_t {
    const UnetLayer &L = u->L[li];
    HW(L.level, H, W);
    return conv3_tc(x->a[coarse], H, W, sh.ch[coarse], u->wpk + u->wpk_off[li], L.cout, x->a[kConvOut[li]],
                    u->status, u->nsm, s, x->a[skip], sh.ch[skip], u->pool);
  };
  auto pool = [&](int src, int dst) {
    HW(sh.lev[src], H, W);
    const size_t n = (size_t)(H / u->pool) * (W / u->pool) * sh.ch[src] / 8;
    return launch_pdl(u->pool == 2 ? k_pool<2> : k_pool<4>, grid_for(n), 256, 0, s, x->a[src], H, W, sh.ch[src],
                      x->a[dst]);
  };
  auto upcat = [&](int coarse, int skip, int dst) {
    HW(sh.lev[skip], H, W);
    const size_t n = (size_t)H * W * sh.ch[dst];
    k_upcat<<<grid_for(n), 256, 0, s>>>(x->a[coarse], sh.ch[coarse], x->a[skip], sh.ch[skip], H, W, u->pool,
                                        x->a[dst]);
    return cudaGetLastError();
  };
  const int skips[3] = {S_E0, S_E1, S_E2}, pooled[3] = {S_P1, S_P2, S_P3};
  for (int l = 0; l < 3; l++) {
    if ((e = conv(2 * l)) || (e = conv(2 * l + 1, pooled[l]))) return e;
    if (!fuse && (e = pool(skips[l], pooled[l]))) return e;
  }
  if ((e = conv(6)) || (e = conv(7))) return e;
  if (fuse) {
    if ((e = conv_cat(8, S_B3, S_E2)) || (e = conv(9))) return e;
    if ((e = conv_cat(10, S_D2, S_E1)) || (e = conv(11))) return e;
    if ((e = conv_cat(12, S_D1, S_E0))) return e;
    const UnetLayer &L = u->L[13];
    return conv3_tc(x->a[S_D0A], u->nr, u->nz, L.cin, u->wpk + u->wpk_off[13], L.cout, keep ? x->a[S_D0] : nullptr,
                    u->status, u->nsm, s, nullptr, 0, 1, ConvEpi{u->wk + u->L[14].woff, u->y, yl, nullptr, 1});
  } else {
    if ((e = upcat(S_B3, S_E2, S_U2)) || (e = conv(8)) || (e = conv(9))) return e;
    if ((e = upcat(S_D2, S_E1, S_U1)) || (e = conv(10)) || (e = conv(11))) return e;
    if ((e = upcat(S_D1, S_E0, S_U0)) || (e = conv(12)) || (e = conv(13))) return e;
  }
  const int P0 = u->nr * u->nz;
  return launch_pdl(k_head, grid_for(P0), 256, 0, s, x->a[S_D0], P0, u->nr, u->ch[0], u->wk + u->L[14].woff, u->y, yl);
}

// backward from u->gy; accumulates parameter gradients into u->gw and, with
// want_dx, the input gradient into ext->gx0
static cudaError_t unet_bwd(const vr_unet *u, bool want_dx, cudaStream_t s) {
  const UnetShapes sh = shapes_of(u);
  const vr_unet *x = u;
  cudaError_t e;
  int H, W;
  auto HW = [&](int lev) {
    H = u->nr;
    W = u->nz;
    for (int l = 0; l < lev; l++) H /= u->pool, W /= u->pool;
  };
  const int P0 = u->nr * u->nz;
  k_head_bwd<<<std::min(P0 / 256 + 1, 148 * 4), 256, 0, s>>>(x->a[S_D0], P0, u->ch[0], u->wk + u->L[14].woff, u->gy,
                                                            x->g[S_D0], u->gw + u->L[14].woff);
  if ((e = cudaGetLastError())) return e;
  // conv layer li: gradient of its output is in g[out]; writes the input
  // gradient to g[in] (or gx0: each has one writer, the skip tensors get their
  // pooling part after it) and adds the weight gradient to gw
  auto conv_bwd = [&](int li, int coarse = -1, int skip = -1) -> cudaError_t {
    const UnetLayer &L = u->L[li];
    HW(L.level);
    const int so = kConvOut[li], si = kConvIn[li];
    const ConvIn in = coarse < 0 ? ConvIn{si < 0 ? u->x0 : x->a[si], L.cin, nullptr, 0, 1}
                                 : ConvIn{x->a[coarse], sh.ch[coarse], x->a[skip], sh.ch[skip], u->pool};
    cudaError_t er = wgrad3(x->g[so], H, W, L.cout, in, L.cin, u->gw + L.woff, u->nsm, s);
    if (er) return er;
    if (si < 0 && !want_dx) return cudaSuccess;
    return dgrad3(x->g[so], H, W, L.cout, u->wk + L.woff, L.cin, si < 0 ? x->gx0 : x->g[si], u->nsm, s);
  };
  auto upcat_bwd = [&](int coarse, int skip, int dst) {
    HW(sh.lev[skip]);
    const size_t n = (size_t)H * W / (u->pool * u->pool) * sh.ch[dst] / 4;
    (u->pool == 2 ? k_upcat_bwd<2> : k_upcat_bwd<4>)<<<grid_for(n), 256, 0, s>>>(
        x->g[dst], sh.ch[coarse], sh.ch[skip], H, W, x->g[coarse], x->g[skip]);
    return cudaGetLastError();
  };
  auto pool_bwd = [&](int src, int dst) {
    HW(sh.lev[src]);
    const size_t n = (size_t)H * W * sh.ch[src] / 4;
    (u->pool == 2 ? k_pool_bwd<2> : k_pool_bwd<4>)<<<grid_for(n), 256, 0, s>>>(x->g[dst], H, W, sh.ch[src], x->g[src]);
    return cudaGetLastError();
  };
  if ((e = conv_bwd(13)) || (e = conv_bwd(12, S_D1, S_E0)) || (e = upcat_bwd(S_D1, S_E0, S_U0))) return e;
  if ((e = conv_bwd(11)) || (e = conv_bwd(10, S_D2, S_E1)) || (e = upcat_bwd(S_D2, S_E1, S_U1))) return e;
  if ((e = conv_bwd(9)) || (e = conv_bwd(8, S_B3, S_E2)) || (e = upcat_bwd(S_B3, S_E2, S_U2))) return e;
  if ((e = conv_bwd(7)) || (e = conv_bwd(6)) || (e = pool_bwd(S_E2, S_P3))) return e;
  if ((e = conv_bwd(5)) || (e = conv_bwd(4)) || (e = pool_bwd(S_E1, S_P2))) return e;
  if ((e = conv_bwd(3)) || (e = conv_bwd(2)) || (e = pool_bwd(S_E0, S_P1))) return e;
  if ((e = conv_bwd(1)) || (e = conv_bwd(0))) return e;
  return cudaSuccess;
}

void unet_dims(const vr_unet *u, int *nr, int *nz) {
  *nr = u->nr;
  *nz = u->nz;
}

cudaError_t unet_read_status(const vr_unet *u, unsigned *st, cudaStream_t s) {
  return cudaMemcpyAsync(st, u->status, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
}
cudaError_t unet_clear_status(const vr_unet *u, cudaStream_t s) {
  return cudaMemsetAsync(u->status, 0, sizeof(unsigned), s);
}

int unet_correct(const vr_unet *u, const double *t, const double *dscale, const double *ss, const int *flags, float *yl,
                 const float **y, cudaStream_t s) {
  const int n = u->nr * u->nz;
  if (launch_pdl(k_in, grid_for(n), 256, 0, s, t, n, ss, 0.0, dscale, u->x0, flags)) return VR_ERR_CUDA;
  if (unet_fwd(u, s, yl, false) != cudaSuccess) return VR_ERR_CUDA;
  *y = u->y;
  return VR_OK;
}

}  // namespace vr

// waits for the stream; reports, once, a tensor-core wait that gave up
static int unet_finish(vr_unet *u) {
  unsigned st = 0;
  U_CUDA(u, unet_read_status(u, &st, u->stream));
  U_CUDA(u, cudaStreamSynchronize(u->stream));
  if (!st) return VR_OK;
  U_CUDA(u, unet_clear_status(u, u->stream));
  U_CUDA(u, cudaStreamSynchronize(u->stream));
  return unet_err(u, VR_ERR_TIMEOUT, "a bounded wait of a convolution gave up");
}

extern "C" int vr_unet_wait_selftest(vr_unet *u, int64_t limit_ns) {
  if (!u || limit_ns < 1000 || limit_ns > 1000000000) return VR_ERR_ARG;
  U_CUDA(u, cudaSetDevice(u->dev));
  U_CUDA(u, launch_wait_selftest((unsigned long long)limit_ns, u->status, u->stream));
  unsigned st = 0;
  U_CUDA(u, unet_read_status(u, &st, u->stream));
  U_CUDA(u, cudaStreamSynchronize(u->stream));
  return st ? VR_ERR_TIMEOUT : VR_OK;
}

extern "C" int vr_unet_forward(vr_unet *u, const double *xh, double *yh) {
  if (!u || !xh || !yh) return VR_ERR_ARG;
  U_CUDA(u, cudaSetDevice(u->dev));
  const int n = u->nr * u->nz;
  double ss = 0.0;
  for (int i = 0; i < n; i++) ss += xh[i] * xh[i];
  const double s = std::sqrt(ss / n);
  U_CUDA(u, cudaMemcpyAsync(u->xs, xh, sizeof(double) * n, cudaMemcpyHostToDevice, u->stream));
  k_in<<<grid_for(n), 256, 0, u->stream>>>(u->xs, n, nullptr, s > 0 ? 1.0 / s : 0.0, nullptr, u->x0, nullptr);
  U_CUDA(u, cudaGetLastError());
  U_CUDA(u, unet_fwd(u, u->stream));
  k_out<<<grid_for(n), 256, 0, u->stream>>>(u->y, n, s, u->xs);
  U_CUDA(u, cudaGetLastError());
  U_CUDA(u, cudaMemcpyAsync(yh, u->xs, sizeof(double) * n, cudaMemcpyDeviceToHost, u->stream));
  return unet_finish(u);
}

__global__ static void k_f2d(const float *a, double *b, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = a[i];
}
__global__ static void k_d2f(const double *a, float *b, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = (float)a[i];
}

extern "C" int vr_unet_backward(vr_unet *u, const double *xh, const double *gh, float *dw, double *dx) {
  if (!u || !xh || !gh) return VR_ERR_ARG;
  U_CUDA(u, cudaSetDevice(u->dev));
  const int n = u->nr * u->nz;
  U_CUDA(u, cudaMemcpyAsync(u->xs, xh, sizeof(double) * n, cudaMemcpyHostToDevice, u->stream));
  k_in<<<grid_for(n), 256, 0, u->stream>>>(u->xs, n, nullptr, 1.0, nullptr, u->x0, nullptr);
  U_CUDA(u, cudaGetLastError());
  U_CUDA(u, unet_fwd(u, u->stream));
  U_CUDA(u, cudaMemcpyAsync(u->xs, gh, sizeof(double) * n, cudaMemcpyHostToDevice, u->stream));
  k_d2f<<<grid_for(n), 256, 0, u->stream>>>(u->xs, u->gy, n);
  U_CUDA(u, cudaMemsetAsync(u->gw, 0, sizeof(float) * u->nparam, u->stream));
  U_CUDA(u, unet_bwd(u, dx != nullptr, u->stream));
  if (dw) U_CUDA(u, cudaMemcpyAsync(dw, u->gw, sizeof(float) * u->nparam, cudaMemcpyDeviceToHost, u->stream));
  if (dx) {
    k_f2d<<<grid_for(n), 256, 0, u->stream>>>(u->gx0, u->xs, n);
    U_CUDA(u, cudaMemcpyAsync(dx, u->xs, sizeof(double) * n, cudaMemcpyDeviceToHost, u->stream));
  }
  return unet_finish(u);
}

extern "C" int vr_unet_train_step(vr_unet *u, vr_k2d *k, const double *e_dev, int32_t nb, float lr, double *loss) {
  if (!u || !k || !e_dev || nb < 1 || !(lr > 0)) return VR_ERR_ARG;
  int32_t knr = 0, knz = 0;
  vr_k2d_info(k, &knr, &knz, nullptr);
  if (knr != u->nr || knz != u->nz) return unet_err(u, VR_ERR_ARG, "network and operator grids differ");
  U_CUDA(u, cudaSetDevice(u->dev));
  const int n = u->nr * u->nz;
  cudaStream_t s = u->stream;
  const double *dh = k2d_dhalf(k);
  U_CUDA(u, cudaMemsetAsync(u->gw, 0, sizeof(float) * u->nparam, s));
  U_CUDA(u, cudaMemsetAsync(u->dscal, 0, sizeof(double) * 8, s));
  for (int b = 0; b < nb; b++) {
    const double *e = e_dev + (size_t)b * n;
    // r = S e; the network sees D r / s (s its RMS), its output maps back as s D yhat
    U_CUDA(u, k2d_train_in(k, e, u->xs, u->dscal + 1, u->dscal + 2, s));
    k_in<<<grid_for(n), 256, 0, s>>>(u->xs, n, u->dscal + 1, 0.0, dh, u->x0, nullptr);
    U_CUDA(u, cudaGetLastError());
    U_CUDA(u, unet_fwd(u, s));
    U_CUDA(u, k2d_train_grad(k, u->y, e, u->xs, u->dscal + 1, u->dscal + 2, u->gy, u->dscal, s));
    U_CUDA(u, unet_bwd(u, false, s));
  }
  // Adam with the batch-mean gradient
  u->adam_t++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, (float)u->adam_t), c2 = 1.f - std::pow(b2, (float)u->adam_t);
  k_adam<<<grid_for(u->nparam), 256, 0, s>>>(u->w32, u->gw, u->m1, u->m2, u->nparam, lr, 1.f / nb, b1, b2, c1, c2,
                                            1e-8f, u->status);
  U_CUDA(u, unet_prep_weights(u, s));
  double h = 0.0;
  U_CUDA(u, cudaMemcpyAsync(&h, u->dscal, sizeof(double), cudaMemcpyDeviceToHost, s));
  const int rc = unet_finish(u);
  if (rc == VR_ERR_TIMEOUT) u->adam_t--;  // no step was made
  if (rc) return rc;
  if (loss) *loss = h / nb;
  return VR_OK;
}
