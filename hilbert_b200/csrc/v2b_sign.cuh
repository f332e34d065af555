// PSD projection of one set of blocks from scratch, without eigenvectors (see
// v2b_sign.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace v2b {

constexpr int kSignSmallDim = 64;   // blocks up to this size: sign_small_kernel
constexpr int kSignSplit = 16;      // CTAs per block in the scaling reductions

// one scaled Newton-Schulz step X <- a X + b X^3
struct SignStep {
    double a, b;
};
// the steps that take every |eigenvalue| from kSignFloor to 1; returns how many
constexpr int kSignMaxSteps = 64;
int sign_steps(SignStep *out /* kSignMaxSteps */);

// blocks of 1 .. kSignSmallDim rows, listed in `list`: x, z from U directly
cudaError_t launch_sign_small(int nlist, const int *list, int max_dim, const double *U, const int64_t *boff,
                              const int *bdim, double inv_mu, double *x, double *z, cudaStream_t s);
// X = Us / ||Us||_F on every listed 64-row tile's block; part: 2 x kSignSplit
// doubles per block
cudaError_t launch_sign_scale(int nblk, int ntiles, const int4 *tiles, const int *bstate, const double *Us,
                              const int64_t *boff, const int *bdim, double *part, double *X, cudaStream_t s);

}  // namespace v2b
