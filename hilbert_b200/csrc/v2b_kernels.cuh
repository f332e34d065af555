// Kernel declarations and launch parameters for the B200 v2RDM path.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "cg_tables.h"
#include "v2b_device.cuh"

namespace v2b {

constexpr int kSpmvThreads = 256;
// One side of the constraint operator as the CG kernel reads it (cg_tables.h)
struct CgRows {
    const uint32_t *off, *ent, *lrp, *lent, *split, *host;
    const uint8_t *len;
    uint32_t nslices, nlong;
};
constexpr int kJacobiThreads = 512;
constexpr int kJacobiMaxDim = 160;     // np*np doubles + rotations must fit in 227 KB
constexpr int kJacobiFoldDim = 80;     // up to here V is rotated beside T: 2 CTAs still fit an SM
constexpr int kStatsBlocks = 256;

struct Palette {
    double v[16];
};

struct CgParams {
    CgRows dual, prim;              // A by constraint, A^T by primal variable
    const uint32_t *orig;           // original row of each dual position
    Palette palA, palT;
    const double *Ax, *Acz, *b;     // rhs = Acz + mu (b - Ax), original order
    double mu;
    double *y;                      // original order, in / out
    double2 *rp;                    // by dual position: the residual and the last direction
    double *yp, *t;                 // by dual and by primal position
    double *slots;                  // 2 x virtual CTAs
    unsigned int *count;            // 0 before the launch
    int *status;
    long long spin_limit;
    double tol;
    int maxit;
    int nvirtual;                   // virtual CTAs, the dot products' partial sums
    double *out;                    // out[0] = iterations, out[1] = final ||r||
    unsigned long long *phase_ns;   // null, or 4 sums of ns: initial residual, pass 1 (A^T p),
                                    // pass 2 (A t and the update), and a slot left at zero
};
// The CG kernel for v = 1, 2 or 3 virtual CTAs to a CTA, one CTA per SM
// (kCgStreamed: v = 1, three CTAs per SM), and its thread count
struct CgShape {
    const void *kernel;
    int threads;
};
CgShape cg_shape(int v, CgTablesIn in);

// Packed rows of A or A^T (CSR) and the list of those longer than
// kSpmvLongRow, which the first long_blocks CTAs take
constexpr uint32_t kSpmvLongRow = 32;
struct SpmvRows {
    const uint32_t *rp, *ent, *long_rows;
    int64_t nrows;
    uint32_t nlong, long_blocks;
};
__global__ void spmv_kernel(SpmvRows R, const double *__restrict__ x, double *__restrict__ y, Palette pal);
__global__ void spmv_A2_kernel(SpmvRows R, const double *__restrict__ x, const double *__restrict__ c,
                               const double *__restrict__ z, double *__restrict__ Ax, double *__restrict__ Acz,
                               Palette pal);
__global__ void spmv_AT_U_kernel(SpmvRows R, const double *__restrict__ y, const double *__restrict__ x,
                                 const double *__restrict__ c, double mu, double *__restrict__ ATy,
                                 double *__restrict__ U, Palette pal);
// the CG starting point of the next outer iteration from the last dual
// solutions (order 0: y itself, 1: 2y - y1, 2: 3y - 3y1 + y2); y1, y2 shift
__global__ void extrapolate_y_kernel(double *__restrict__ y, double *__restrict__ y1,
                                     double *__restrict__ y2, int64_t n, int order);
__global__ void stats_kernel(const double *__restrict__ Ax, const double *__restrict__ b,
                             const double *__restrict__ ATy, const double *__restrict__ z,
                             const double *__restrict__ c, const double *__restrict__ x,
                             const double *__restrict__ y, int64_t np, int64_t nd,
                             double *__restrict__ partials, unsigned int *counter,
                             double *__restrict__ out, int *status);
__global__ void jacobi_warm_kernel(const double *__restrict__ T0, double *__restrict__ Pout,
                                   double *__restrict__ Vt, const int64_t *__restrict__ boff,
                                   const int *__restrict__ bdim, double2 *__restrict__ rot,
                                   const int64_t *__restrict__ rot_off, int max_sweeps,
                                   double abs_tol, double gap_tol, int *status, int *rot_count,
                                   int raw = 0);
__global__ void identity_blocks_kernel(double *__restrict__ Vt, const int64_t *__restrict__ boff,
                                       const int *__restrict__ bdim);
__global__ void half_residual_kernel(const double *__restrict__ G, double *__restrict__ H,
                                     const int64_t *__restrict__ boff, const int *__restrict__ bdim);

// Raise func's dynamic shared-memory limit on the current device to at least
// bytes, under one process-wide lock; never lowers it, because several
// problems (and the allocation-free entry point) share the attribute.
cudaError_t raise_dynamic_smem(const void *func, int bytes);
// Unique id of the current CUDA context, 0 when there is none.  A new
// context (after cudaDeviceReset) gets a new id, so per-device caches of
// symbol addresses and function attributes can tell that they are stale.
unsigned long long current_context_id();

inline size_t jacobi_smem_bytes(int n) {
    const int np = n + (n & 1);
    // T with odd rows (columns free of bank conflicts); V beside it up to
    // kJacobiFoldDim rows; monotone in n, so that the largest block's size serves all
    const size_t one = (size_t)np * (np + 1) * sizeof(double);
    constexpr size_t fold = 2 * (size_t)kJacobiFoldDim * (kJacobiFoldDim + 1) * sizeof(double);
    const size_t mats = n <= kJacobiFoldDim ? 2 * one : (one > fold ? one : fold);
    return mats + (size_t)(np / 2) * (sizeof(double2) + sizeof(int));
}

}  // namespace v2b
