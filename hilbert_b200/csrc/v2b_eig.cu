// Batched FP64 GEMM tiles for the warm-started PSD projection (sm_100a).
//
// Between outer iterations U = mu x + A^T y - c changes little, so the
// eigenvectors of the previous iteration (rows of Vt) nearly diagonalise the
// new block: per iteration
//   W  = sym(U) Vt^T          gemm<N,T>
//   T0 = Vt W                 gemm<N,N>      (= V^T U V, nearly diagonal)
//   selective Jacobi on T0    jacobi_warm_kernel (shared memory, one CTA per block)
//   Y  = Vt^T P               gemm<T,N>
//   U+ = Y Vt                 gemm<N,N> with the projection epilogue
//                             x = U+ / mu,  z = U+ - sym(U)
// Every gemm launch covers all blocks of the problem: its work is the list of
// output tiles (64 x 64 or 32 x 32) of every block.
#include "v2b_eig.cuh"
#include "v2b_kernels.cuh"

#include <mutex>

#include <algorithm>

namespace v2b {

// ---------------------------------------------------------------------------
// batched FP64 GEMM over square blocks: C_b = op(A_b) op(B_b) [+ epilogue]
//
// FP64 tensor cores (mma.sync m8n8k4 .f64): a 64 x 64 output tile per CTA of
// 4 warps, each warp a 32 x 32 sub-tile of 4 x 4 m8n8 fragments (32
// accumulators per thread); a 32 x 32 tile has a quarter of each.  K runs in
// chunks of 16 through a cp.async pipeline of three stages, six for the smaller
// tile (8-byte copies: a block of odd dimension starts at an
// odd double, so 16-byte alignment is not available; out-of-range elements
// are zero-filled by the copy itself).  Each operand tile is stored with its
// global contiguous index innermost (k-major when the matrix is read down
// its columns), padded so that both the copies and the fragment reads are
// free of bank conflicts.
//
// With a scheduler counter the grid is persistent (the SM count times the
// CTAs an SM holds) and CTAs take tiles in list order, the tile list sorted
// by block dimension (its K) descending: the longest tiles start first and
// the short ones fill in behind them.  Without one, CTA i computes tile i.
//
// Split K: when a launch has fewer tiles than the grid has CTA slots, the
// plan cuts the K range of the large blocks' tiles into S parts (tile word w:
// bit 0 mirror, bit 1 only the upper half of a diagonal tile, bits 4-7 the part s, bits 8-11 S, bits 12+ the output tile's
// group; S <= kGemmMaxSplit).  Each part stores its 64 x 64 partial product
// in the group's slot s of split_ws and counts itself in split_cnt[group]; the part that arrives
// last sums the slots in the order s = 0 .. S-1 (the same bits whichever
// part arrives last), re-arms the counter and runs the epilogue.
//
// Tile size: 64 x 64 tiles reuse their operands twice as often, 32 x 32 tiles
// (a quarter of the work, 0.14 us of MMAs per K chunk against 0.54) give four
// times as many CTAs and finish sooner where 64 x 64 tiles leave SMs idle.  A
// warm projection pair and a stand-alone projection, us with 32 / 64: 6 orbitals
// 418 / 552 and 857 / 1,650, 9: 649 / 943 and 1,026 / 2,056, 11: 744 / 1,091 and
// 1,224 / 2,534, 5 with T2: 568 / 999 and 1,060 / 2,126.
constexpr int kGemmBK = 16;
constexpr int kGemmThreads = 128;
constexpr int kPadK = kGemmBK + 4;      // m-major rows: 16 + 4 doubles
template <int TM>
struct GemmShape {
    static constexpr int kPadM = TM + 4;   // k-major rows
    static constexpr int kOpDoubles = (TM * kPadK > kGemmBK * kPadM) ? TM * kPadK : kGemmBK * kPadM;
    // the K chunks of a 32-row tile are short: more of them in flight
    static constexpr int kStages = TM == 64 ? 3 : 6;
    static constexpr int kSmem = kStages * 2 * kOpDoubles * (int)sizeof(double);
};

__device__ __forceinline__ void cp_async8(double *smem, const double *gmem, bool pred) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    const int bytes = pred ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// D (8 x 8) += A (8 x 4, row) B (4 x 8, col); per lane: A[l/4][l%4],
// B[l%4][l/4], D[l/4][2 (l%4) + {0, 1}]
__device__ __forceinline__ void dmma_8x8x4(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// shared-memory index of element (m, k) of a TM x 16 operand tile
template <int TM, bool KMAJOR>
__device__ __forceinline__ int op_idx(int m, int k) {
    return KMAJOR ? k * GemmShape<TM>::kPadM + m : m * kPadK + k;
}

// one TM x 16 operand tile: rows m of the operand (rows of op(A) or columns of
// op(B)) from m0, k from k0.  KMAJOR: the global matrix is contiguous in m
// (element (m, k) at X[k n + m]), else in k (X[m n + k]).
template <int TM, bool KMAJOR>
__device__ __forceinline__ void load_op(double *sm, const double *__restrict__ X, int n, int m0, int k0) {
#pragma unroll
    for (int it = 0; it < TM * kGemmBK / kGemmThreads; it++) {
        const int e = it * kGemmThreads + threadIdx.x;
        const int m = KMAJOR ? e % TM : e / kGemmBK;
        const int k = KMAJOR ? e / TM : e % kGemmBK;
        const int gm = m0 + m, gk = k0 + k;
        const bool ok = gm < n && gk < n;
        const double *src = ok ? (KMAJOR ? X + (int64_t)gk * n + gm : X + (int64_t)gm * n + gk) : X;
        cp_async8(sm + op_idx<TM, KMAJOR>(m, k), src, ok);
    }
}

template <int TM, bool TA, bool TB, int EPI>
__global__ void __launch_bounds__(kGemmThreads, 3)
    gemm_tiles_kernel(const double *__restrict__ A, const double *__restrict__ B,
                      double *__restrict__ C, const int4 *__restrict__ tiles,
                      const int64_t *__restrict__ boff, const int *__restrict__ bdim,
                      const double *__restrict__ Cin, const double *__restrict__ Us, double inv_mu, double beta,
                      double *__restrict__ xo, double *__restrict__ zo,
                      const int *__restrict__ bstate, unsigned long long *__restrict__ orth,
                      int ntiles, int *__restrict__ sched, double *__restrict__ split_ws,
                      int *__restrict__ split_cnt) {
    // op(A) rows are m-contiguous in memory when A is read transposed;
    // op(B) columns are m-contiguous when B is read as stored
    constexpr bool AK = TA, BKM = !TB;
    constexpr int kGemmStages = GemmShape<TM>::kStages;
    constexpr int kOpDoubles = GemmShape<TM>::kOpDoubles, F = TM / 16;   // F x F fragments per warp
    extern __shared__ double gsm[];
    __shared__ int s_tile, s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = (warp >> 1) * (TM / 2), wn = (warp & 1) * (TM / 2);
    const int fr = lane >> 2, fk = lane & 3;
    for (int iter = 0;; iter++) {
        int ti;
        if (sched) {
            if (threadIdx.x == 0) {
                int t = atomicAdd(sched, 1);
                if (t >= ntiles) {
                    // the last CTA to run out re-arms the counter for the next launch
                    if (atomicAdd(sched + 1, 1) == (int)gridDim.x - 1) {
                        sched[0] = 0;
                        sched[1] = 0;
                    }
                    t = -1;
                }
                s_tile = t;
            }
            __syncthreads();
            ti = s_tile;
            __syncthreads();
        } else {
            ti = iter == 0 ? (int)blockIdx.x : -1;
        }
        if (ti < 0) break;
        const int4 t = tiles[ti];
        const int blk = t.x, n = bdim[blk];
        if (bstate && bstate[blk] != 0) continue;   // uniform over the CTA
        const int64_t off = boff[blk];
        const int r0 = t.y * TM, c0 = t.z * TM;
        const double *Ab = A + off, *Bb = B + off;
        double acc[F][F][2];
#pragma unroll
        for (int i = 0; i < F; i++)
#pragma unroll
            for (int j = 0; j < F; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

        const int split = (t.w >> 8) & 15, part = (t.w >> 4) & 15;
        const int nk_all = (n + kGemmBK - 1) / kGemmBK;
        // this part's K chunks: kb .. kb + nk - 1
        const int per = split > 1 ? (nk_all + split - 1) / split : nk_all;
        const int kb = split > 1 ? min(part * per, nk_all) : 0;
        const int nk = min(nk_all - kb, per);
#pragma unroll
        for (int st = 0; st < kGemmStages - 1; st++) {
            if (st < nk) {
                double *sa = gsm + st * 2 * kOpDoubles;
                load_op<TM, AK>(sa, Ab, n, r0, (kb + st) * kGemmBK);
                load_op<TM, BKM>(sa + kOpDoubles, Bb, n, c0, (kb + st) * kGemmBK);
            }
            cp_async_commit();
        }
        for (int kt = 0; kt < nk; kt++) {
            cp_async_wait<kGemmStages - 2>();
            __syncthreads();
            // refill the stage consumed one step ago (every warp is past it)
            const int kn = kt + kGemmStages - 1;
            if (kn < nk) {
                double *sa = gsm + (kn % kGemmStages) * 2 * kOpDoubles;
                load_op<TM, AK>(sa, Ab, n, r0, (kb + kn) * kGemmBK);
                load_op<TM, BKM>(sa + kOpDoubles, Bb, n, c0, (kb + kn) * kGemmBK);
            }
            cp_async_commit();
            const double *sa = gsm + (kt % kGemmStages) * 2 * kOpDoubles;
            const double *sb = sa + kOpDoubles;
#pragma unroll
            for (int k4 = 0; k4 < kGemmBK; k4 += 4) {
                double a[F], b[F];
#pragma unroll
                for (int i = 0; i < F; i++) a[i] = sa[op_idx<TM, AK>(wm + i * 8 + fr, k4 + fk)];
#pragma unroll
                for (int j = 0; j < F; j++) b[j] = sb[op_idx<TM, BKM>(wn + j * 8 + fr, k4 + fk)];
#pragma unroll
                for (int i = 0; i < F; i++)
#pragma unroll
                    for (int j = 0; j < F; j++) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
            }
        }
        cp_async_wait<0>();
        __syncthreads();   // the next tile's copies reuse the stages

        if (split > 1) {
            const unsigned group = (unsigned)t.w >> 12;
            double *slot = split_ws + ((int64_t)group * kGemmMaxSplit + part) * (TM * TM);
#pragma unroll
            for (int i = 0; i < F; i++)
#pragma unroll
                for (int j = 0; j < F; j++)
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        __stcg(slot + (wm + i * 8 + fr) * TM + wn + j * 8 + 2 * fk + h, acc[i][j][h]);
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) s_last = atomicAdd(split_cnt + group, 1) == split - 1;
            __syncthreads();
            if (!s_last) continue;
            __threadfence();
            const double *slots = split_ws + (int64_t)group * kGemmMaxSplit * (TM * TM);
#pragma unroll
            for (int i = 0; i < F; i++)
#pragma unroll
                for (int j = 0; j < F; j++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int e = (wm + i * 8 + fr) * TM + wn + j * 8 + 2 * fk + h;
                        double v = __ldcg(slots + e);
                        for (int q = 1; q < split; q++) v += __ldcg(slots + q * (TM * TM) + e);
                        acc[i][j][h] = v;
                    }
            if (threadIdx.x == 0) split_cnt[group] = 0;   // every part has arrived: re-arm
        }

        double dev = 0.0;
#pragma unroll
        for (int i = 0; i < F; i++) {
            const int r = r0 + wm + i * 8 + fr;
            if (r >= n) continue;
#pragma unroll
            for (int j = 0; j < F; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int c = c0 + wn + j * 8 + 2 * fk + h;
                    if (c >= n) continue;
                    if ((t.w & 2) && c < r) continue;   // a strictly symmetric result's diagonal tile
                    const double v = acc[i][j][h];
                    // t.w: an off-diagonal tile of a symmetric product, stored
                    // at (r, c) and at its mirror image (c, r)
                    for (int m = 0; m <= (t.w & 1); m++) {
                        const int64_t e = m ? off + (int64_t)c * n + r : off + (int64_t)r * n + c;
                        if (EPI == kEpiStore) {
                            C[e] = v;
                        } else if (EPI == kEpiAdd) {
                            C[e] = Cin[e] + v;
                        } else if (EPI == kEpiNS) {   // v = (Vt Vt^T)[r][c]
                            const double id = (r == c) ? 1.0 : 0.0;
                            C[e] = 1.5 * id - 0.5 * v;
                            dev = fmax(dev, fabs(v - id));
                        } else if (EPI == kEpiLinear) {
                            C[e] = inv_mu * Cin[e] + beta * v;
                        } else if (EPI == kEpiSign) {   // v = Us sign(Us)
                            const double up = 0.5 * (Us[e] + v);
                            xo[e] = up * inv_mu;
                            zo[e] = up - Us[e];
                        } else {   // kEpiProject: v = U+
                            xo[e] = v * inv_mu;
                            zo[e] = v - Us[e];
                        }
                    }
                }
        }
        if (EPI == kEpiNS) {
            // non-negative doubles order like their bit patterns
            dev = warp_max(dev);
            if (lane == 0 && dev > 0.0)
                atomicMax(orth + blk, (unsigned long long)__double_as_longlong(dev));
        }
    }
}

template <int TM, bool TA, bool TB, int EPI>
static cudaError_t launch_variant(int ntiles, cudaStream_t s, GEMM_ARGS, int *sched, double *split_ws,
                                  int *split_cnt, double beta) {
    auto kern = gemm_tiles_kernel<TM, TA, TB, EPI>;
    constexpr int kGemmSmem = GemmShape<TM>::kSmem;
    // opt in to the pipeline's shared memory and size the persistent grid,
    // once per variant, device and context (function attributes are per
    // device and do not survive a cudaDeviceReset)
    struct Cfg {
        unsigned long long ctx = 0;
        int slots = 0;
    };
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static Cfg cache[kMaxDevices];
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    Cfg cfg;
    {
        std::lock_guard<std::mutex> lock(mu);
        const unsigned long long ctx = current_context_id();
        if (cache[dev].slots == 0 || cache[dev].ctx != ctx) {
            int sms = 0, occ = 0;
            err = raise_dynamic_smem((const void *)kern, kGemmSmem);
            if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (err == cudaSuccess)
                err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kGemmThreads, kGemmSmem);
            if (err != cudaSuccess) return err;
            // the context id is read after the calls above, which create the context if needed
            cache[dev].ctx = current_context_id();
            cache[dev].slots = std::max(1, sms * occ);
        }
        cfg = cache[dev];
    }
    const int grid = sched ? std::min(ntiles, cfg.slots) : ntiles;
    kern<<<grid, kGemmThreads, kGemmSmem, s>>>(A, B, C, tiles, boff, bdim, Cin, Us, inv_mu, beta, xo, zo,
                                               bstate, orth, ntiles, sched, split_ws, split_cnt);
    return cudaGetLastError();
}

cudaError_t launch_gemm_tiles(GemmVariant v, int ntiles, cudaStream_t s, GEMM_ARGS, int *sched, double *split_ws,
                              int *split_cnt, int tile, double beta) {
    if (ntiles <= 0) return cudaSuccess;
#define V2B_GEMM_CASE(NAME, TA, TB, EPI)                                                                            \
    case NAME:                                                                                                      \
        return tile == 32 ? launch_variant<32, TA, TB, EPI>(ntiles, s, A, B, C, tiles, boff, bdim, Cin, Us, inv_mu, \
                                                            xo, zo, bstate, orth, sched, split_ws, split_cnt, beta)  \
                          : launch_variant<64, TA, TB, EPI>(ntiles, s, A, B, C, tiles, boff, bdim, Cin, Us, inv_mu, \
                                                            xo, zo, bstate, orth, sched, split_ws, split_cnt, beta);
    switch (v) {
        V2B_GEMM_CASE(kGemmNTNewtonSchulz, false, true, kEpiNS)
        V2B_GEMM_CASE(kGemmNTStore, false, true, kEpiStore)
        V2B_GEMM_CASE(kGemmNNStore, false, false, kEpiStore)
        V2B_GEMM_CASE(kGemmTNStore, true, false, kEpiStore)
        V2B_GEMM_CASE(kGemmNNProject, false, false, kEpiProject)
        V2B_GEMM_CASE(kGemmNNAdd, false, false, kEpiAdd)
        V2B_GEMM_CASE(kGemmNTLinear, false, true, kEpiLinear)
        V2B_GEMM_CASE(kGemmNTSign, false, true, kEpiSign)
    }
#undef V2B_GEMM_CASE
    return cudaErrorInvalidValue;
}

// Us = (U + U^T) / 2 per block, tile by tile
__global__ void symmetrize_kernel(const double *__restrict__ U, double *__restrict__ Us,
                                  const int4 *__restrict__ tiles, const int64_t *__restrict__ boff,
                                  const int *__restrict__ bdim) {
    const int4 t = tiles[blockIdx.x];
    const int n = bdim[t.x];
    const int64_t off = boff[t.x];
    for (int e = threadIdx.x; e < 64 * 64; e += blockDim.x) {
        const int r = t.y * 64 + e / 64, c = t.z * 64 + e % 64;
        if (r < n && c < n)
            Us[off + (int64_t)r * n + c] = 0.5 * (U[off + (int64_t)r * n + c] + U[off + (int64_t)c * n + r]);
    }
}

}  // namespace v2b
