// PSD projection without eigenvectors: U+ = (U + U sign(U)) / 2 (sm_100a).
//
// A stand-alone projection keeps no basis for a next one, so it needs the
// projector only, not the eigenvectors: sign(U) from the Newton-Schulz
// iteration X <- 3/2 (r X) - 1/2 (r X)^3 of X0 = sym(U) / ||U||_F, with the
// scaling r = sqrt(3 / (1 + l + l^2)) that maps [l, 1] best (Chen and Chow,
// "A stable scaling of Newton-Schulz for improving the sign function
// computation of a Hermitian matrix", 2014), capped at kSignMaxScale: the cap
// keeps the image of 1 above 0.2, without which rounding errors of the large
// eigenvalues grow with the small ones.  Every step is two products of
// symmetric matrices that commute, so half of each is computed and mirrored:
// 2 x 43 half products on FP64 tensor cores and no host decision, against
// Jacobi sweeps whose rotations are a serial chain.  Blocks of 11 to 242 rows
// ((11e,11o) DQG): 1.2 ms against 15.4 ms.
//
// An eigenvalue below kSignFloor ||U||_F may keep a factor in (-1, 1) instead
// of its sign: an error of at most half of it.  Against 64-bit references the
// result is 1e-15 .. 3e-15 ||U+||_F off for spectra with gaps, degenerate and
// rank-deficient ones and ones spread over 16 decades (the Jacobi path: 1e-13).
#include "v2b_sign.cuh"

#include <algorithm>
#include <cmath>

#include "v2b_kernels.cuh"

namespace v2b {

constexpr double kSignFloor = 1e-15;
constexpr double kSignMaxScale = 1.65;

int sign_steps(SignStep *out) {
    double l = kSignFloor;
    int n = 0;
    while (1.0 - l > 1e-15 && n < kSignMaxSteps) {
        const double r = std::min(kSignMaxScale, std::sqrt(3.0 / (1.0 + l + l * l)));
        out[n++] = SignStep{1.5 * r, -0.5 * r * r * r};
        // the least of the image of [l, 1]: at l, or at 1 under the cap
        const double at_l = l * (1.5 * r - 0.5 * r * r * r * l * l), at_1 = 1.5 * r - 0.5 * r * r * r;
        l = std::min(at_l, at_1);
    }
    return n;
}

// ------------------------------------------------------------ small blocks
// One CTA per block: Us, X and Y in shared memory.  The upper 8 x 8 tiles of a
// product are dealt to the eight warps, up to five to a warp, whose chains of
// m8n8k4 MMAs hide each other's latency; a symmetric operand is read by rows
// for either side.
constexpr int kSignTiles = 5;   // ceil(36 / 8)
constexpr int kSignThreads = 256;

struct SignSteps {
    int n;
    SignStep s[kSignMaxSteps];
};

__global__ void __launch_bounds__(kSignThreads)
    sign_small_kernel(const int *__restrict__ list, const double *__restrict__ U, const int64_t *__restrict__ boff,
                      const int *__restrict__ bdim, double inv_mu, double *__restrict__ x, double *__restrict__ z,
                      SignSteps steps) {
    const int blk = list[blockIdx.x], n = bdim[blk];
    const int64_t off = boff[blk];
    const int nt = (n + 7) / 8, np = 8 * nt, ntri = nt * (nt + 1) / 2;
    const int ld = np + 4;
    extern __shared__ double sm[];
    double *S = sm, *X = S + np * ld, *Y = X + np * ld;
    __shared__ double red[32], s_scale;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int fr = lane >> 2, fk = lane & 3;
    const double *Ub = U + off;
    double big = 0.0;
    for (int e = tid; e < np * np; e += kSignThreads) {
        const int i = e / np, j = e % np;
        const double v = i < n && j < n ? 0.5 * (Ub[(int64_t)i * n + j] + Ub[(int64_t)j * n + i]) : 0.0;
        S[i * ld + j] = v;
        big = fmax(big, fabs(v));
    }
    big = block_max(big, red);
    if (tid == 0) s_scale = big;
    __syncthreads();
    big = s_scale;
    double fro = 0.0;
    if (big > 0.0)
        for (int e = tid; e < np * np; e += kSignThreads) {
            const double v = S[e / np * ld + e % np] / big;
            fro = fma(v, v, fro);
        }
    fro = block_sum(fro, red);
    if (tid == 0) s_scale = fro;
    __syncthreads();
    const double norm = sqrt(s_scale);
    // a NaN anywhere in the block (fmax passes over it) reaches every element
    for (int e = tid; e < np * np; e += kSignThreads) {
        const double v = S[e / np * ld + e % np];
        X[e / np * ld + e % np] = big > 0.0 ? v / big / norm : v;
    }
    // this warp's tiles (tr <= tc)
    int tr[kSignTiles], tc[kSignTiles];
#pragma unroll
    for (int q = 0; q < kSignTiles; q++) {
        const int t = warp + 8 * q;
        int r = 0, left = t;
        while (r < nt && left >= nt - r) {
            left -= nt - r;
            r++;
        }
        tr[q] = t < ntri ? r : -1;
        tc[q] = t < ntri ? r + left : 0;
    }
    const int mine = ntri > warp ? (ntri - warp + 7) / 8 : 0;
    double c[kSignTiles][2];
    // c = the tiles of A B for symmetric commuting A, B
    auto product = [&](const double *A, const double *B) {
#pragma unroll
        for (int q = 0; q < kSignTiles; q++) c[q][0] = c[q][1] = 0.0;
        for (int k = 0; k < np; k += 4)
#pragma unroll
            for (int q = 0; q < kSignTiles; q++)
                if (q < mine) {
                    const double a = A[(8 * tr[q] + fr) * ld + k + fk], b = B[(8 * tc[q] + fr) * ld + k + fk];
                    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                                 : "+d"(c[q][0]), "+d"(c[q][1])
                                 : "d"(a), "d"(b));
                }
    };
    // each element of the tiles and its mirror image
    auto store = [&](double *D, auto &&f) {
#pragma unroll
        for (int q = 0; q < kSignTiles; q++)
            if (q < mine)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int r = 8 * tr[q] + fr, cc = 8 * tc[q] + 2 * fk + h;
                    if (tr[q] == tc[q] && cc < r) continue;   // the diagonal tile's upper half
                    const double v = f(r, cc, c[q][h]);
                    D[r * ld + cc] = v;
                    D[cc * ld + r] = v;
                }
    };
    __syncthreads();
    for (int k = 0; k < steps.n; k++) {
        product(X, X);
        store(Y, [](int, int, double v) { return v; });
        __syncthreads();
        product(X, Y);
        __syncthreads();   // X has been read
        const SignStep st = steps.s[k];
        store(X, [&](int r, int cc, double v) { return fma(st.b, v, st.a * X[r * ld + cc]); });
        __syncthreads();
    }
    product(S, X);
    store(Y, [&](int r, int cc, double v) { return 0.5 * (S[r * ld + cc] + v); });   // U+
    __syncthreads();
    for (int e = tid; e < n * n; e += kSignThreads) {
        const int i = e / n, j = e % n;
        const double up = Y[i * ld + j];
        x[off + e] = up * inv_mu;
        z[off + e] = up - S[i * ld + j];
    }
}

cudaError_t launch_sign_small(int nlist, const int *list, int max_dim, const double *U, const int64_t *boff,
                              const int *bdim, double inv_mu, double *x, double *z, cudaStream_t s) {
    if (nlist <= 0) return cudaSuccess;
    static const SignSteps steps = [] {
        SignSteps q;
        q.n = sign_steps(q.s);
        return q;
    }();
    const int np = (max_dim + 7) & ~7;
    const int smem = 3 * np * (np + 4) * (int)sizeof(double);
    const cudaError_t e = raise_dynamic_smem((const void *)sign_small_kernel, smem);
    if (e != cudaSuccess) return e;
    sign_small_kernel<<<nlist, kSignThreads, smem, s>>>(list, U, boff, bdim, inv_mu, x, z, steps);
    return cudaGetLastError();
}

// ------------------------------------------------------------ larger blocks
// scaling in two reductions over kSignSplit CTAs a block (largest magnitude,
// then the norm of the block over it: no overflow), in a fixed order
__global__ void __launch_bounds__(256)
    sign_max_kernel(const double *__restrict__ Us, const int64_t *__restrict__ boff, const int *__restrict__ bdim,
                    const int *__restrict__ bstate, double *__restrict__ part) {
    const int blk = blockIdx.x;
    if (bstate[blk] != 0) return;
    const int64_t nn = (int64_t)bdim[blk] * bdim[blk];
    __shared__ double red[32];
    double v = 0.0;
    for (int64_t e = (int64_t)blockIdx.y * 256 + threadIdx.x; e < nn; e += 256 * kSignSplit)
        v = fmax(v, fabs(Us[boff[blk] + e]));
    v = block_max(v, red);
    if (threadIdx.x == 0) part[(size_t)blk * 2 * kSignSplit + blockIdx.y] = v;
}
__device__ __forceinline__ double sign_big(const double *part, int blk) {
    double big = 0.0;
    for (int k = 0; k < kSignSplit; k++) big = fmax(big, part[(size_t)blk * 2 * kSignSplit + k]);
    return big;
}
__global__ void __launch_bounds__(256)
    sign_norm_kernel(const double *__restrict__ Us, const int64_t *__restrict__ boff, const int *__restrict__ bdim,
                     const int *__restrict__ bstate, double *__restrict__ part) {
    const int blk = blockIdx.x;
    if (bstate[blk] != 0) return;
    const int64_t nn = (int64_t)bdim[blk] * bdim[blk];
    __shared__ double red[32];
    const double big = sign_big(part, blk);
    double v = 0.0;
    if (big > 0.0)
        for (int64_t e = (int64_t)blockIdx.y * 256 + threadIdx.x; e < nn; e += 256 * kSignSplit) {
            const double u = Us[boff[blk] + e] / big;
            v = fma(u, u, v);
        }
    v = block_sum(v, red);
    if (threadIdx.x == 0) part[(size_t)blk * 2 * kSignSplit + kSignSplit + blockIdx.y] = v;
}
__global__ void __launch_bounds__(256)
    sign_scale_kernel(const double *__restrict__ Us, const int4 *__restrict__ tiles, const int64_t *__restrict__ boff,
                      const int *__restrict__ bdim, const int *__restrict__ bstate, const double *__restrict__ part,
                      double *__restrict__ X) {
    const int4 t = tiles[blockIdx.x];
    if (bstate[t.x] != 0) return;
    const int n = bdim[t.x];
    const int64_t off = boff[t.x];
    const double big = sign_big(part, t.x);
    double sum = 0.0;
    for (int k = 0; k < kSignSplit; k++) sum += part[(size_t)t.x * 2 * kSignSplit + kSignSplit + k];
    const double norm = sqrt(sum);
    for (int e = threadIdx.x; e < 64 * 64; e += 256) {
        const int r = t.y * 64 + e / 64, c = t.z * 64 + e % 64;
        if (r >= n || c >= n) continue;
        const double v = Us[off + (int64_t)r * n + c];
        X[off + (int64_t)r * n + c] = big > 0.0 ? v / big / norm : v;
    }
}

cudaError_t launch_sign_scale(int nblk, int ntiles, const int4 *tiles, const int *bstate, const double *Us,
                              const int64_t *boff, const int *bdim, double *part, double *X, cudaStream_t s) {
    sign_max_kernel<<<dim3(nblk, kSignSplit), 256, 0, s>>>(Us, boff, bdim, bstate, part);
    sign_norm_kernel<<<dim3(nblk, kSignSplit), 256, 0, s>>>(Us, boff, bdim, bstate, part);
    sign_scale_kernel<<<ntiles, 256, 0, s>>>(Us, tiles, boff, bdim, bstate, part, X);
    return cudaGetLastError();
}

}  // namespace v2b
