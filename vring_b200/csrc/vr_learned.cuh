// vr_learned.cuh -- internal interface between the Krylov solvers
// (vr_krylov.cu) and the learned preconditioner (vr_unet.cu).
#pragma once

#include <cuda_runtime.h>

#include "../../include/vring_b200.h"

namespace vr {

// y = N(D t / s), D = dscale (per cell) and s = sqrt(*ss / n) with
// ss = sum (D t)^2 read on the device; t a device array of nr*nz doubles, *y
// the network's own output array, yl (may be null) a copy of its last radial
// row (nz values).  The input is left alone once flags[0] is set.
int unet_correct(const vr_unet *u, const double *t, const double *dscale, const double *ss, const int *flags, float *yl,
                 const float **y, cudaStream_t s);

// A solver holds the network that it is given: its captured iterations have the
// network's buffers in them.  A destroyed network's memory, and with it its
// address, is free for another one only after the last holder has dropped it.
void unet_hold(const vr_unet *u);
void unet_drop(const vr_unet *u);

// the word that a convolution sets when its bounded tensor-core wait gives up
// (its outputs are then not valid); the caller synchronises the stream
cudaError_t unet_read_status(const vr_unet *u, unsigned *st, cudaStream_t s);
cudaError_t unet_clear_status(const vr_unet *u, cudaStream_t s);

// grid of a network (nr, nz)
void unet_dims(const vr_unet *u, int *nr, int *nz);

// D^-1/2 of the symmetric operator's diagonal, per cell (device)
const double *k2d_dhalf(const vr_k2d *k);

// Training pair of one sample: r = S e, ss = sum (D r)^2, er = e . r
// (device scalars); r a device array of nr*nz
cudaError_t k2d_train_in(vr_k2d *k, const double *e, double *r, double *ss, double *er, cudaStream_t s);
// Energy-norm loss of the network output yhat (float) for the pair (e, r):
//   y = s D yhat, res = S y - r, loss_acc += (y - e) . res / er,
//   gyhat = 2 s D res / er  (the gradient of the loss with respect to yhat)
cudaError_t k2d_train_grad(vr_k2d *k, const float *yhat, const double *e, const double *r, const double *ss,
                           const double *er, float *gyhat, double *loss_acc, cudaStream_t s);

}  // namespace vr
