// CUDA kernels of the B200 boundary-point iteration (sm_100a).
//
//   spmv_kernel          y = A.x or A^T.y over packed rows (bit-exact to hilbert's maps)
//   spmv_A2_kernel       A.x and A.(c - z) in one pass over A's rows
//   spmv_AT_U_kernel     A^T.y and U = mu x + A^T y - c in one pass over A^T's rows
//   cg_kernel            persistent conjugate-gradient solve of (A A^T) y = rhs
//   stats_kernel         eps_p^2, eps_d^2, c.x, b.y (deterministic reductions)
//   jacobi_warm_kernel   per-block selective Jacobi on V^T U V in shared memory,
//                        middle factor of U+ and the refined eigenvectors
#include "v2b_kernels.cuh"

#include <cuda.h>

#include <mutex>

namespace v2b {

// ---------------------------------------------------------------- maps
// A x and A^T y in hilbert's order: a row's products (one multiply rounding
// each) are added left to right, entries from the first flagged one on in a
// second sum.  Most rows hold one to three entries, a thread each, kRowBatch
// entries' operands in flight; the few long ones (traces, contractions: up to
// 400 entries at (20e,20o)) would each hold a thread for as many dependent
// additions behind loads, so they go to a warp each, first in the grid: the
// lanes fetch and multiply 128 entries at a time, one lane per sum adds them
// in order from shared memory.
//
// Measured on B200, (20e,20o), A x and A^T y together: 60 us (a thread for
// every row: 124).
constexpr int kRowBatch = 4;
constexpr int kSpmvWarps = kSpmvThreads / 32;
constexpr int kLongChunk = 128;

struct OneVector {
    static constexpr int N = 1;
    const double *x;
    __device__ __forceinline__ void get(uint32_t c, double (&v)[1]) const { v[0] = __ldg(x + c); }
};
struct XAndCz {   // x and c - z
    static constexpr int N = 2;
    const double *x, *c, *z;
    __device__ __forceinline__ void get(uint32_t k, double (&v)[2]) const {
        v[0] = __ldg(x + k);
        v[1] = __dsub_rn(__ldg(c + k), __ldg(z + k));
    }
};

// out(row, sums) for every row
template <class X, class F>
__device__ __forceinline__ void row_sums(const SpmvRows &R, const X &x, const double *pal, F &&out) {
    constexpr int N = X::N;
    __shared__ double buf[kSpmvWarps][N][kLongChunk];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x < R.long_blocks) {
        const uint32_t q = blockIdx.x * kSpmvWarps + warp;
        if (q >= R.nlong) return;
        const uint32_t r = __ldg(R.long_rows + q), b = __ldg(R.rp + r), e = __ldg(R.rp + r + 1);
        double acc0 = 0.0, acc1 = 0.0;
        bool grp = false;
        for (uint32_t k0 = b; k0 < e; k0 += kLongChunk) {
            const int cnt = (int)min((uint32_t)kLongChunk, e - k0);
            uint32_t w[kLongChunk / 32];
            double v[kLongChunk / 32][N];
#pragma unroll
            for (int i = 0; i < kLongChunk / 32; i++) w[i] = 32 * i + lane < cnt ? __ldg(R.ent + k0 + 32 * i + lane) : 0u;
#pragma unroll
            for (int i = 0; i < kLongChunk / 32; i++) x.get(w[i] & kDevColMask, v[i]);
            int first = cnt;   // the first flagged entry of the chunk
#pragma unroll
            for (int i = kLongChunk / 32 - 1; i >= 0; i--) {
                const unsigned m = __ballot_sync(0xffffffffu, w[i] >> 31);
                if (m) first = 32 * i + __ffs(m) - 1;
#pragma unroll
                for (int n = 0; n < N; n++) buf[warp][n][32 * i + lane] = __dmul_rn(pal[(w[i] >> 27) & 15u], v[i][n]);
            }
            __syncwarp();
            if (lane < N) {
                const int split = grp ? 0 : first;
#pragma unroll 8
                for (int i = 0; i < split; i++) acc0 = __dadd_rn(acc0, buf[warp][lane][i]);
#pragma unroll 8
                for (int i = split; i < cnt; i++) acc1 = __dadd_rn(acc1, buf[warp][lane][i]);
            }
            grp = grp || first < cnt;
            __syncwarp();
        }
        double s[N];
        const double mine = grp ? __dadd_rn(acc0, acc1) : acc0;
#pragma unroll
        for (int n = 0; n < N; n++) s[n] = __shfl_sync(0xffffffffu, mine, n);
        if (lane == 0) out((int64_t)r, s);
        return;
    }
    for (int64_t r = (int64_t)(blockIdx.x - R.long_blocks) * blockDim.x + threadIdx.x; r < R.nrows;
         r += (int64_t)(gridDim.x - R.long_blocks) * blockDim.x) {
        const uint32_t b = __ldg(R.rp + r), e = __ldg(R.rp + r + 1);
        if (e - b > kSpmvLongRow) continue;
        double acc0[N] = {}, acc1[N] = {};
        bool grp = false;
        for (uint32_t k0 = b; k0 < e; k0 += kRowBatch) {
            uint32_t w[kRowBatch];
            double v[kRowBatch][N];
#pragma unroll
            for (int i = 0; i < kRowBatch; i++) w[i] = k0 + i < e ? __ldg(R.ent + k0 + i) : 0u;
#pragma unroll
            for (int i = 0; i < kRowBatch; i++)
                if (k0 + i < e) x.get(w[i] & kDevColMask, v[i]);
#pragma unroll
            for (int i = 0; i < kRowBatch; i++) {
                if (k0 + i >= e) continue;
                grp = grp || (w[i] >> 31);
#pragma unroll
                for (int n = 0; n < N; n++) {
                    const double u = __dmul_rn(pal[(w[i] >> 27) & 15u], v[i][n]);
                    if (grp) acc1[n] = __dadd_rn(acc1[n], u);
                    else acc0[n] = __dadd_rn(acc0[n], u);
                }
            }
        }
        double s[N];
#pragma unroll
        for (int n = 0; n < N; n++) s[n] = grp ? __dadd_rn(acc0[n], acc1[n]) : acc0[n];
        out(r, s);
    }
}

__global__ void __launch_bounds__(kSpmvThreads)
    spmv_kernel(SpmvRows R, const double *__restrict__ x, double *__restrict__ y, Palette pal) {
    __shared__ double spal[16];
    if (threadIdx.x < 16) spal[threadIdx.x] = pal.v[threadIdx.x];
    __syncthreads();
    row_sums(R, OneVector{x}, spal, [&](int64_t r, const double (&s)[1]) { y[r] = s[0]; });
}

__global__ void __launch_bounds__(kSpmvThreads)
    spmv_A2_kernel(SpmvRows R, const double *__restrict__ x, const double *__restrict__ c,
                   const double *__restrict__ z, double *__restrict__ Ax, double *__restrict__ Acz, Palette pal) {
    __shared__ double spal[16];
    if (threadIdx.x < 16) spal[threadIdx.x] = pal.v[threadIdx.x];
    __syncthreads();
    row_sums(R, XAndCz{x, c, z}, spal, [&](int64_t r, const double (&s)[2]) {
        Ax[r] = s[0];
        Acz[r] = s[1];
    });
}

__global__ void __launch_bounds__(kSpmvThreads)
    spmv_AT_U_kernel(SpmvRows R, const double *__restrict__ y, const double *__restrict__ x,
                     const double *__restrict__ c, double mu, double *__restrict__ ATy, double *__restrict__ U,
                     Palette pal) {
    __shared__ double spal[16];
    if (threadIdx.x < 16) spal[threadIdx.x] = pal.v[threadIdx.x];
    __syncthreads();
    row_sums(R, OneVector{y}, spal, [&](int64_t r, const double (&s)[1]) {
        const double a = s[0];
        ATy[r] = a;
        U[r] = mu * x[r] + a - c[r];
    });
}

// ------------------------------------------------------------------ CG
// Solves (A A^T) y = rhs with rhs = A(c - z) + mu (b - A x), warm-started from
// y, in the form CG takes on normal equations: with t = A^T p the step
// length's denominator p.(A A^T p) is ||t||^2, which the pass that forms t
// sums as it goes.  Two grid barriers per iteration, each carrying its sum:
//   1. t = A^T p with p = r + beta p_old formed per operand from the pair
//      (r, p_old), partial ||t||^2                      -> alpha = r.r / ||t||^2
//   2. per constraint j: q = (A t)_j, p_j again from its pair, y_j += alpha
//      p_j, r_j -= alpha q, partial r.r                  -> beta, convergence
// r and p_old are one 16-byte pair, so an operand costs one gather; p is never
// read by another row in pass 2, so pass 2 replaces the pair in place.
//
// Rounding: products and sums are those of the stored order of each row
// (separate multiply and add), the dot products those of the virtual CTAs
// (cg_tables.h): 16 warps with one accumulator per lane, a shuffle tree per
// warp, one per CTA, one over the CTAs.  The iteration count of a solve hangs
// on the last bits (the residual meets the tolerance on a plateau), so the
// order is part of the result; a CTA hosts V virtual CTAs, and NW warps share
// their 16 V virtual warps.
//
// What bounds it: dependent loads (entry, then operand) and the two barriers,
// with all tables and vectors in L2; so a warp has several slices' loads in
// flight, and one CTA per SM meets at the barrier.

// the operand p (PAIR: r + beta p_old of a pair; else a plain vector)
template <bool PAIR>
struct Operand {
    const double2 *rp;
    const double *x;
    double beta;
    __device__ __forceinline__ double operator()(uint32_t pos) const {
        if (!PAIR) return x[pos];
        const double2 v = rp[pos];
        return __dadd_rn(v.x, __dmul_rn(beta, v.y));
    }
};

// a compile-time count
template <int K>
struct Count {
    __device__ constexpr operator int() const { return K; }
};
// table words in shared memory, or streamed through L2 without displacing the
// vectors
template <bool SMEM>
struct Words {
    const uint32_t *p;
    __device__ __forceinline__ uint32_t operator[](uint32_t k) const { return SMEM ? p[k] : __ldcs(p + k); }
    __device__ __forceinline__ Words operator+(uint32_t k) const { return Words{p + k}; }
};

// the lane's row of one slice: entries in stored order, separate multiply and
// add, flagged entries in a second sum; STEP operands in flight (the loads are
// unconditional, from position 0 past a row's end, so that none waits for
// another).  SELF: entries at kCgSelf take coef * self instead.
template <int STEP, bool SELF, bool SMEM, class X>
__device__ __forceinline__ double sell_row(const Words<SMEM> &ent, uint32_t width, uint32_t len, const X &x, double self,
                                           const double *pal) {
    double acc0 = 0.0, acc1 = 0.0;
    bool grp = false;
    for (uint32_t k0 = 0; k0 < width; k0 += STEP) {
        uint32_t w[STEP];
        double v[STEP];
#pragma unroll
        for (int k = 0; k < STEP; k++) w[k] = k0 + k < len ? ent[32u * (k0 + k)] : 0u;
#pragma unroll
        for (int k = 0; k < STEP; k++) {
            const uint32_t c = w[k] & kDevColMask;
            v[k] = x(SELF && c == kCgSelf ? 0u : c);
        }
#pragma unroll
        for (int k = 0; k < STEP; k++) {
            const double cf = pal[(w[k] >> 27) & 15u];
            const double u = __dmul_rn(cf, SELF && (w[k] & kDevColMask) == kCgSelf ? __dmul_rn(cf, self) : v[k]);
            const bool in = k0 + k < len;
            grp = grp || (in && (w[k] >> 31));
            const double s0 = __dadd_rn(acc0, u), s1 = __dadd_rn(acc1, u);
            acc0 = in && !grp ? s0 : acc0;
            acc1 = in && grp ? s1 : acc1;
        }
    }
    return grp ? __dadd_rn(acc0, acc1) : acc0;
}
// a long row by one warp: the lanes stride over the entries, a shuffle tree
template <class X>
__device__ __forceinline__ double warp_row(const uint32_t *ent, uint32_t b, uint32_t e, const X &x, const double *pal,
                                           int lane) {
    double acc = 0.0;
    for (uint32_t k0 = b; k0 < e; k0 += 128) {
        uint32_t w[4];
        double v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) w[k] = k0 + 32u * k + lane < e ? ent[k0 + 32u * k + lane] : 0u;
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = x(w[k] & kDevColMask);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (k0 + 32u * k + lane < e) acc += pal[(w[k] >> 27) & 15u] * v[k];
    }
    return warp_sum(acc);
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// V virtual CTAs to a CTA of NW warps; U plain slices and STEP operands of
// another row in flight.  A virtual warp's tables (a few KB) are always read
// from shared memory: a table word read from L2 would put one more dependent
// load before every operand (12 joint rings: 24 us per iteration against 40).
// Where the SM holds both passes' tables they are copied once (kCgBoth); else
// the two passes share the region, and each warp starts the copy of the next
// pass's tables as it ends a pass, so that it runs behind the barrier
// (kCgOneRegion); tables too large for that are streamed from L2 and HBM
// (kCgStreamed: evict first, the vectors stay in L2).
template <int NW, int V, int U, int STEP, int CTAS, CgTablesIn IN>
__global__ void __launch_bounds__(32 * NW, CTAS) cg_kernel(CgParams P) {
    constexpr int VW = kCgVirtualWarps * V;    // virtual warps of a full CTA
    constexpr int H = VW / NW;                 // per warp
    constexpr bool SMEM = IN != kCgStreamed, SHARED = IN == kCgOneRegion;
    static_assert(H * NW == VW, "whole virtual warps");
    extern __shared__ __align__(16) uint32_t cg_sm[];
    __shared__ double palA[16], palT[16];
    __shared__ double red[VW], total;
    __shared__ int fail;
    __shared__ unsigned long long tmark;   // phase clock (CTA 0, thread 0)
    __shared__ uint32_t hostA[V], hostT[V];
    __shared__ CgRun runA[VW], runT[VW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cta = blockIdx.x;
    if (tid < 16) {
        palA[tid] = P.palA.v[tid];
        palT[tid] = P.palT.v[tid];
    }
    if (tid == 0) fail = 0;
    if (tid < V) {
        hostA[tid] = P.dual.host[cta * V + tid];
        hostT[tid] = P.prim.host[cta * V + tid];
    }
    const uint32_t all = (uint32_t)P.nvirtual * kCgVirtualWarps;
    __syncthreads();
    auto words = [&](const CgRows &R, const CgRun &r) {
        return r.gw == 0xffffffffu ? 0u
                                   : cg_table_words(r.e - r.b, (R.off[r.e] & ~kCgPlain) - (R.off[r.b] & ~kCgPlain));
    };
    if (tid < VW) {
        auto init = [&](CgRun &r, const CgRows &R, uint32_t vc) {
            r = CgRun{0u, 0u, 0xffffffffu, 0u, 0, 0u};
            if (vc == 0xffffffffu) return;
            r.gw = vc * kCgVirtualWarps + tid % kCgVirtualWarps;
            r.b = R.split[r.gw];
            r.e = R.split[r.gw + 1];
        };
        init(runA[tid], P.dual, hostA[tid / kCgVirtualWarps]);
        init(runT[tid], P.prim, hostT[tid / kCgVirtualWarps]);
        runA[tid].off = words(P.dual, runA[tid]);
        runT[tid].off = words(P.prim, runT[tid]);
    }
    __syncthreads();
    if (SMEM && tid == 0) {   // where each run's tables go
        uint32_t at = 0;
        for (int w = 0; w < VW; w++) {
            const uint32_t na = runA[w].off, nt = runT[w].off;
            runA[w].ent = (int32_t)at;
            runT[w].ent = (int32_t)(SHARED ? at : at + na);
            at += SHARED ? max(na, nt) : na + nt;
        }
    }
    __syncthreads();
    // start the copy of a run's tables: entries, lengths, offsets
    auto fetch = [&](const CgRows &R, const CgRun &r) {
        if (r.gw == 0xffffffffu) return;
        const uint32_t e0 = R.off[r.b] & ~kCgPlain, ne = (R.off[r.e] & ~kCgPlain) - e0, n = r.e - r.b;
        const uint32_t at = (uint32_t)r.ent + e0;   // the word of entry e0
        for (uint32_t k = 4u * lane; k < ne; k += 128u) cp_async16(cg_sm + at + k, R.ent + e0 + k);
        for (uint32_t k = lane; k < 2u * n; k += 32u)
            cp_async16((uint8_t *)cg_sm + r.len + 16u * k, R.len + 32u * (size_t)r.b + 16u * k);
        for (uint32_t k = lane; k <= n; k += 32u) cp_async4(cg_sm + r.off + k, R.off + r.b + k);
    };
    if (SMEM && tid < VW) {
        auto place = [&](CgRun &r, const CgRows &R) {
            if (r.gw == 0xffffffffu) return;
            const uint32_t e0 = R.off[r.b] & ~kCgPlain, ne = (R.off[r.e] & ~kCgPlain) - e0;
            cg_place_run(r, (uint32_t)r.ent, e0, ne);
        };
        place(runA[tid], P.dual);
        place(runT[tid], P.prim);
    }
    const uint32_t dl = 32u * P.dual.nslices, tl = 32u * P.prim.nslices;   // positions of the long rows
    GridSum bar{P.slots, P.nvirtual, P.count, P.status, P.spin_limit, &total, &fail, 0u};
    // barrier + sum of one value per lane of every virtual warp
    auto sync = [&](const double (&loc)[H], const uint32_t *host, double &sum) {
#pragma unroll
        for (int h = 0; h < H; h++) {
            const double w = warp_sum(loc[h]);
            if (lane == 0) red[warp + h * NW] = w;
        }
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int v = 0; v < V; v++) {
                double s = lane < kCgVirtualWarps ? red[v * kCgVirtualWarps + lane] : 0.0;
                s = warp_sum(s);
                if (lane == 0 && host[v] != 0xffffffffu) __stcg(bar.set() + host[v], s);
            }
            bar.arrive_and_sum(lane);
        }
        __syncthreads();
        return bar.done(sum);
    };
    if (tid == 0) tmark = global_ns();
    __syncthreads();
    // tables of the pass ahead (SHARED), or of both passes once
    auto fetch_T = [&](bool start) {
        if (!SMEM || (!SHARED && !start)) return;
        __syncwarp();
#pragma unroll
        for (int h = 0; h < H; h++) fetch(P.prim, runT[warp + h * NW]);
    };
    auto fetch_A = [&](bool start) {
        if (!SMEM || (!SHARED && !start)) return;
        __syncwarp();
#pragma unroll
        for (int h = 0; h < H; h++) fetch(P.dual, runA[warp + h * NW]);
    };
    auto fetched = [&]() {
        if (!SMEM) return;
        cp_async_wait_all();
        __syncwarp();
    };
    fetch_T(true);
    if (!SHARED) fetch_A(true);
    auto lap = [&](int k) {   // optional phase clock: CTA 0 adds the time from barrier to barrier
        if (P.phase_ns != nullptr && cta == 0 && tid == 0) {
            const unsigned long long now = global_ns();
            P.phase_ns[k] += now - tmark;
            tmark = now;
        }
    };
    // t = A^T x over a run's slices: stored except at singles, squares into
    // loc in order (loc null: no squares)
    auto apply_T = [&](const CgRun &r, const auto &x, double *loc) {
        const uint32_t e = r.e;
        const Words<SMEM> ent{SMEM ? cg_sm + r.ent + lane : P.prim.ent + lane};
        const Words<SMEM> off{SMEM ? cg_sm + r.off - r.b : P.prim.off};
        const uint8_t *len = SMEM ? (const uint8_t *)cg_sm + r.len - 32 * (size_t)r.b + lane : P.prim.len + lane;
        // K plain slices from s on
        auto plain = [&](auto K, const uint32_t *o) {
            uint32_t w[K];
            double v[K];
#pragma unroll
            for (int u = 0; u < K; u++) w[u] = ent[o[u] & ~kCgPlain];
#pragma unroll
            for (int u = 0; u < K; u++) v[u] = x(w[u] & kDevColMask);
            if (loc)
#pragma unroll
                for (int u = 0; u < K; u++) {
                    const double tv = __dmul_rn(palT[w[u] >> 27], v[u]);
                    *loc = fma(tv, tv, *loc);
                }
        };
        for (uint32_t s = r.b; s < e;) {
            uint32_t o[U];
            bool all_plain = s + U <= e;
#pragma unroll
            for (int u = 0; u < U; u++) {
                o[u] = off[min(s + u, e)];
                all_plain = all_plain && (o[u] & kCgPlain);
            }
            if (all_plain) {
                plain(Count<U>(), o);
                s += U;
                continue;
            }
            if (o[0] & kCgPlain) {
                plain(Count<1>(), o);
                s++;
                continue;
            }
            const uint32_t n = len[32u * s], o1 = off[s + 1] & ~kCgPlain, width = (o1 - o[0]) >> 5;
            if (n != kCgPadding) {
                const double tv = width <= 2 ? sell_row<2, false, SMEM>(ent + o[0], width, n & 0x7fu, x, 0.0, palT)
                                             : sell_row<STEP, false, SMEM>(ent + o[0], width, n & 0x7fu, x, 0.0, palT);
                if (!(n & kCgSingle)) P.t[32u * s + lane] = tv;
                if (loc) *loc = fma(tv, tv, *loc);
            }
            s++;
        }
    };
    auto long_T = [&](uint32_t gw, const auto &x, double *loc) {
        for (uint32_t l = gw; l < P.prim.nlong; l += all) {
            const double v = warp_row(P.prim.lent, P.prim.lrp[l], P.prim.lrp[l + 1], x, palT, lane);
            if (lane == 0) {
                P.t[tl + l] = v;
                if (loc) *loc = fma(v, v, *loc);
            }
        }
    };
    // f(position, (A t) there, own) over a run's slices, in order; own =
    // own0(position) is loaded with the entries, self(own) is the p that the
    // row's singles take
    const Operand<false> tx{nullptr, P.t, 0.0};
    auto apply_A = [&](const CgRun &r, auto &&own0, auto &&self, auto &&f) {
        const uint32_t e = r.e;
        const Words<SMEM> ent{SMEM ? cg_sm + r.ent + lane : P.dual.ent + lane};
        const Words<SMEM> off{SMEM ? cg_sm + r.off - r.b : P.dual.off};
        const uint8_t *len = SMEM ? (const uint8_t *)cg_sm + r.len - 32 * (size_t)r.b + lane : P.dual.len + lane;
        auto plain = [&](auto K, uint32_t s, const uint32_t *o) {
            uint32_t w[K][2];
            double v[K][2];
            decltype(own0(0u)) own[K];
#pragma unroll
            for (int u = 0; u < K; u++) {
                own[u] = own0(32u * (s + u) + lane);
                w[u][0] = ent[o[u] & ~kCgPlain];
                w[u][1] = ent[(o[u] & ~kCgPlain) + 32u];
            }
#pragma unroll
            for (int u = 0; u < K; u++)
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const uint32_t c = w[u][k] & kDevColMask;
                    v[u][k] = P.t[c == kCgSelf ? 0u : c];
                }
#pragma unroll
            for (int u = 0; u < K; u++) {
                const double sv = self(own[u]);
                double q[2];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const double c = palA[w[u][k] >> 27];
                    q[k] = __dmul_rn(c, (w[u][k] & kDevColMask) == kCgSelf ? __dmul_rn(c, sv) : v[u][k]);
                }
                f(32u * (s + u) + lane, __dadd_rn(q[0], q[1]), own[u]);
            }
        };
        for (uint32_t s = r.b; s < e;) {
            uint32_t o[U];
            bool all_plain = s + U <= e;
#pragma unroll
            for (int u = 0; u < U; u++) {
                o[u] = off[min(s + u, e)];
                all_plain = all_plain && (o[u] & kCgPlain);
            }
            if (all_plain) {
                plain(Count<U>(), s, o);
                s += U;
                continue;
            }
            if (o[0] & kCgPlain) {
                plain(Count<1>(), s, o);
                s++;
                continue;
            }
            const uint32_t n = len[32u * s], o1 = off[s + 1] & ~kCgPlain, width = (o1 - o[0]) >> 5;
            if (n != kCgPadding) {
                const auto own = own0(32u * s + lane);
                const double q = width <= 2 ? sell_row<2, true, SMEM>(ent + o[0], width, n, tx, self(own), palA)
                                            : sell_row<(STEP < 8 ? STEP : 8), true, SMEM>(ent + o[0], width, n, tx,
                                                                                          self(own), palA);
                f(32u * s + lane, q, own);
            }
            s++;
        }
    };
    auto long_A = [&](uint32_t gw, auto &&own0, auto &&f) {
        for (uint32_t l = gw; l < P.dual.nlong; l += all) {
            const double v = warp_row(P.dual.lent, P.dual.lrp[l], P.dual.lrp[l + 1], tx, palA, lane);
            if (lane == 0) f(dl + l, v, own0(dl + l));
        }
    };
    // copy(original row, position) over the own constraints, C at a time
    constexpr int C = 4;
    auto own_rows = [&](auto &&load, auto &&store) {
#pragma unroll
        for (int h = 0; h < H; h++) {
            const CgRun &r = runA[warp + h * NW];
            if (r.gw == 0xffffffffu) continue;
            for (uint32_t s = r.b; s < r.e; s += C) {
                uint32_t o[C];
                double v[C];
#pragma unroll
                for (int u = 0; u < C; u++) o[u] = s + u < r.e ? P.orig[32u * (s + u) + lane] : 0xffffffffu;
#pragma unroll
                for (int u = 0; u < C; u++) v[u] = o[u] != 0xffffffffu ? load(o[u], 32u * (s + u) + lane) : 0.0;
#pragma unroll
                for (int u = 0; u < C; u++)
                    if (o[u] != 0xffffffffu) store(o[u], 32u * (s + u) + lane, v[u]);
            }
            if (lane == 0)
                for (uint32_t l = r.gw; l < P.dual.nlong; l += all)
                    store(P.orig[dl + l], dl + l, load(P.orig[dl + l], dl + l));
        }
    };

    // r = rhs - A A^T y
    double zero[H] = {}, loc[H], sum, rs;
    own_rows([&](uint32_t o, uint32_t) { return P.y[o]; }, [&](uint32_t, uint32_t j, double v) { P.yp[j] = v; });
    auto stopped = [&]() {   // no copy may be in flight when a CTA leaves
        cp_async_wait_all();
    };
    if (!sync(zero, hostA, sum)) return stopped();
    fetched();
    {
        const Operand<false> yx{nullptr, P.yp, 0.0};
#pragma unroll
        for (int h = 0; h < H; h++) {
            const CgRun &r = runT[warp + h * NW];
            if (r.gw == 0xffffffffu) continue;
            apply_T(r, yx, nullptr);
            long_T(r.gw, yx, nullptr);
        }
    }
    fetch_A(false);
    if (!sync(zero, hostA, sum)) return stopped();
    fetched();
    {
        struct Own {
            double y, acz, b, ax;
        };
        auto own0 = [&](uint32_t j) {
            const uint32_t o = P.orig[j];
            return Own{P.yp[j], P.Acz[o], P.b[o], P.Ax[o]};
        };
#pragma unroll
        for (int h = 0; h < H; h++) {
            loc[h] = 0.0;
            const CgRun &r = runA[warp + h * NW];
            if (r.gw == 0xffffffffu) continue;
            auto f = [&](uint32_t j, double av, const Own &o) {
                const double v = o.acz + P.mu * (o.b - o.ax) - av;
                P.rp[j] = make_double2(v, 0.0);
                loc[h] = fma(v, v, loc[h]);
            };
            apply_A(r, own0, [](const Own &o) { return o.y; }, f);
            long_A(r.gw, own0, f);
        }
    }
    fetch_T(false);
    if (!sync(loc, hostA, rs)) return stopped();
    lap(0);

    int it = 0;
    double beta = 0.0;
    bool done = !(sqrt(rs) >= P.tol);
    while (!done && it < P.maxit) {
        // pass 1
        fetched();
        const Operand<true> px{P.rp, nullptr, beta};
#pragma unroll
        for (int h = 0; h < H; h++) {
            loc[h] = 0.0;
            const CgRun &r = runT[warp + h * NW];
            if (r.gw == 0xffffffffu) continue;
            apply_T(r, px, &loc[h]);
            long_T(r.gw, px, &loc[h]);
        }
        fetch_A(false);
        double tt;
        if (!sync(loc, hostT, tt)) break;
        lap(1);
        if (!(tt > 0.0)) break;   // range of A A^T exhausted (or non-finite)
        const double alpha = rs / tt;

        // pass 2
        fetched();
        struct Own {
            double2 rp;
            double y;
        };
        auto own0 = [&](uint32_t j) { return Own{P.rp[j], P.yp[j]}; };
        auto dir = [&](const Own &o) { return __dadd_rn(o.rp.x, __dmul_rn(beta, o.rp.y)); };
#pragma unroll
        for (int h = 0; h < H; h++) {
            loc[h] = 0.0;
            const CgRun &r = runA[warp + h * NW];
            if (r.gw == 0xffffffffu) continue;
            auto f = [&](uint32_t j, double q, const Own &o) {
                const double pn = dir(o);
                P.yp[j] = fma(alpha, pn, o.y);
                const double rv = fma(-alpha, q, o.rp.x);
                P.rp[j] = make_double2(rv, pn);
                loc[h] = fma(rv, rv, loc[h]);
            };
            long_A(r.gw, own0, f);
            apply_A(r, own0, dir, f);
        }
        fetch_T(false);
        double rs_new;
        if (!sync(loc, hostA, rs_new)) break;
        lap(2);
        it++;
        if (!(rs_new == rs_new)) {   // NaN
            if (cta == 0 && tid == 0) atomicExch(P.status, kStatusNan);
            break;
        }
        done = sqrt(rs_new) < P.tol;
        beta = rs_new / rs;
        rs = rs_new;
    }
    cp_async_wait_all();   // the tables of a pass that does not come
    if (fail) return;
    own_rows([&](uint32_t, uint32_t j) { return P.yp[j]; }, [&](uint32_t o, uint32_t, double v) { P.y[o] = v; });
    if (cta == 0 && tid == 0) {
        P.out[0] = (double)it;
        P.out[1] = sqrt(rs);
    }
}

// Measured on B200 (us per CG iteration; in brackets the former kernel: two
// gathers per operand, tables read from L2, three CTAs of 512 threads per SM,
// a barrier of three round trips):
//   6-site ring 7.4 (22.9), (9e,9o) 11.5 (30), (6e,6o) DQGT2 12.9 (31),
//   DOCI (10e,10o) 6.6 (15.9), 12 joint rings 18.1 (48), (20e,20o) 47 (84).
// Warps and operands in flight, same order: a warp per virtual warp where one
// or two virtual CTAs share an SM ((9e,9o), 16 warps: 12.0); three on 24 warps
// (on 16 warps (20e,20o) took 53, as three CTAs of 16 warps 64).
CgShape cg_shape(int v, CgTablesIn in) {
    if (in == kCgStreamed) return {(const void *)cg_kernel<16, 1, 2, 4, 3, kCgStreamed>, 512};
    if (v == 1) return {(const void *)cg_kernel<16, 1, 1, 8, 1, kCgBoth>, 512};
    if (v == 2) return {(const void *)cg_kernel<32, 2, 1, 8, 1, kCgBoth>, 1024};
    if (in == kCgBoth) return {(const void *)cg_kernel<24, 3, 2, 8, 1, kCgBoth>, 768};
    return {(const void *)cg_kernel<24, 3, 2, 4, 1, kCgOneRegion>, 768};
}

// ------------------------------------------------------- CG start
// The dual solution moves smoothly from one outer iteration to the next
// while mu stays fixed, so the conjugate gradients start from its polynomial
// extrapolation through the last solutions (linear after one, quadratic
// after two) instead of the last one.  The CG still runs to the same
// residual tolerance: only the number of its iterations changes (about half
// on the benchmark problems, the same outer iterations and energies to
// 1e-8 Eh).
__global__ void extrapolate_y_kernel(double *__restrict__ y, double *__restrict__ y1,
                                     double *__restrict__ y2, int64_t n, int order) {
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
        const double v = y[j], v1 = y1[j];
        if (order == 1) y[j] = 2.0 * v - v1;
        else if (order == 2) y[j] = 3.0 * (v - v1) + y2[j];
        y2[j] = v1;
        y1[j] = v;
    }
}

// --------------------------------------------------------------- stats
// out[0] = ||A x - b||^2, out[1] = ||A^T y + z - c||^2, out[2] = c.x, out[3] = b.y
__global__ void stats_kernel(const double *__restrict__ Ax, const double *__restrict__ b,
                             const double *__restrict__ ATy, const double *__restrict__ z,
                             const double *__restrict__ c, const double *__restrict__ x,
                             const double *__restrict__ y, int64_t np, int64_t nd,
                             double *__restrict__ partials, unsigned int *counter,
                             double *__restrict__ out, int *status) {
    __shared__ double red[32];
    __shared__ bool last;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // kBatch elements' loads in flight; each sum keeps its order
    constexpr int kBatch = 4;
    for (int64_t j0 = gtid; j0 < nd; j0 += kBatch * stride) {
        double va[kBatch], vb[kBatch], vy[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int64_t j = j0 + u * stride;
            va[u] = j < nd ? Ax[j] : 0.0;
            vb[u] = j < nd ? b[j] : 0.0;
            vy[u] = j < nd ? y[j] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kBatch; u++)
            if (j0 + u * stride < nd) {
                const double d = va[u] - vb[u];
                s[0] += d * d;
                s[3] += vb[u] * vy[u];
            }
    }
    for (int64_t i0 = gtid; i0 < np; i0 += kBatch * stride) {
        double va[kBatch], vz[kBatch], vc[kBatch], vx[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int64_t i = i0 + u * stride;
            va[u] = i < np ? ATy[i] : 0.0;
            vz[u] = i < np ? z[i] : 0.0;
            vc[u] = i < np ? c[i] : 0.0;
            vx[u] = i < np ? x[i] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kBatch; u++)
            if (i0 + u * stride < np) {
                const double d = va[u] + vz[u] - vc[u];
                s[1] += d * d;
                s[2] += vc[u] * vx[u];
            }
    }
    for (int k = 0; k < 4; k++) {
        const double v = block_sum(s[k], red);
        if (threadIdx.x == 0) partials[k * gridDim.x + blockIdx.x] = v;
    }
    __threadfence();
    if (threadIdx.x == 0) last = (atomicAdd(counter, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int k = 0; k < 4; k++) {
        double v = 0.0;
        if (threadIdx.x < 32) {
            for (int i = threadIdx.x; i < (int)gridDim.x; i += 32)
                v += *((volatile double *)(partials + k * gridDim.x + i));
            v = warp_sum(v);
        }
        if (threadIdx.x == 0) {
            out[k] = v;
            if (!(v == v) || v - v != 0.0) atomicExch(status, kStatusNan);
        }
    }
    if (threadIdx.x == 0) *counter = 0u;
}

// --------------------------------------------------------- projection

// One CTA per PSD block (n <= kJacobiMaxDim): selective parallel cyclic
// Jacobi on T = V^T U V, where the rows of Vt (= V^T) are the previous
// iteration's eigenvectors (the identity on a cold start).
//
// A pair (p, q) is rotated (sym.schur2, Golub & Van Loan sec. 8.5) only when
// the first-order (Daleckii-Krein) projection formula could not settle it:
//     t_pq^2 > gap_tol * ||T||_F * |t_pp - t_qq|   and   |t_pq| > abs_tol * ||T||_F.
// Sweeps repeat until a sweep rotates nothing.  The kernel then writes the
// middle factor of U+ = V P V^T,
//     P_ii = max(t_ii, 0),   P_ij = t_ij (t_ii+ - t_jj+) / (t_ii - t_jj)   (i != j),
// (with raw != 0: the rotated T itself, for callers that want eigenvalues)
// and rotates Vt likewise (rows p, q of Vt per rotation), leaving the refined
// eigenvectors for the next iteration: up to kJacobiFoldDim rows Vt lies in
// shared memory beside T and takes each step's rotations with it; above, T's
// rotations are recorded and replayed on Vt once T has made room for it.
//
// Bound by latency: a step is a chain of square roots and divisions, then two
// barriers; a warp takes a pair row P, its lanes the columns, and skips the row
// if nothing rotates it.  One nearly diagonal block of 10, 24, 64, 160 rows: 29,
// 80, 363, 3,126 us; with a list of the rotated pairs made between two more
// barriers, rows of even length and a replay for every block 40, 102, 573,
// 5,817 us.  Fewer threads are no faster on small blocks (10 rows: 29 us with
// 256, 35 with 128).
__global__ void __launch_bounds__(kJacobiThreads)
    jacobi_warm_kernel(const double *__restrict__ T0, double *__restrict__ Pout,
                       double *__restrict__ Vt, const int64_t *__restrict__ boff,
                       const int *__restrict__ bdim, double2 *__restrict__ rot,
                       const int64_t *__restrict__ rot_off, int max_sweeps, double abs_tol,
                       double gap_tol, int *status, int *rot_count, int raw) {
    extern __shared__ double sm[];
    const int blk = blockIdx.x;
    const int n = bdim[blk];
    if (n <= 0) return;
    const int64_t off = boff[blk];
    const int np = n + (n & 1);
    const int m = np / 2;
    const int ld = np + 1;
    const bool fold = n <= kJacobiFoldDim;
    double *T = sm;                      // np x ld
    double *V = fold ? T + (size_t)np * ld : T;   // np x ld, rows = eigenvectors
    double2 *cs = (double2 *)(V + (size_t)np * ld);   // m
    int *act = (int *)(cs + m);          // m
    __shared__ double red[32];
    __shared__ double s_nrm;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    double *Vb = Vt + off;
    auto load_V = [&]() {
        for (int i = warp; i < np; i += warps)
            for (int j = lane; j < np; j += 32)
                V[i * ld + j] = (i < n && j < n) ? Vb[(int64_t)i * n + j] : (i == j ? 1.0 : 0.0);
    };
    // rows p, q of V by the rotations of step st in cs, act
    auto rotate_V = [&](int st) {
        for (int P = warp; P < m; P += warps) {
            if (!act[P]) continue;
            const double2 r = cs[P];
            int p, q;
            rr_pair(st, P, np, p, q);
            for (int j = lane; j < np; j += 32) {
                const double vp = V[p * ld + j], vq = V[q * ld + j];
                V[p * ld + j] = r.x * vp - r.y * vq;
                V[q * ld + j] = r.y * vp + r.x * vq;
            }
        }
    };

    const double *Tb = T0 + off;
    double fro = 0.0;
    for (int e = threadIdx.x; e < np * np; e += blockDim.x) {
        const int i = e / np, j = e % np;
        double v = 0.0;
        if (i < n && j < n) v = 0.5 * (Tb[(int64_t)i * n + j] + Tb[(int64_t)j * n + i]);
        T[i * ld + j] = v;
        fro += v * v;
    }
    if (fold) load_V();
    fro = block_sum(fro, red);
    if (threadIdx.x == 0) s_nrm = sqrt(fro);
    __syncthreads();
    const double nrm = s_nrm;
    const double atol = abs_tol * nrm + 1e-300, gtol = gap_tol * nrm;

    double2 *rb = rot + rot_off[blk];
    int sweep = 0, total = 0, nrot = 0;   // the same on every thread
    for (; sweep < max_sweeps; sweep++) {
        nrot = 0;
        for (int st = 0; st < np - 1; st++) {
            const int k = threadIdx.x;   // blockDim.x >= m: a thread a pair
            int a = 0;
            if (k < m) {
                int p, q;
                rr_pair(st, k, np, p, q);
                double c = 1.0, s = 0.0;
                if (q < n) {
                    const double apq = T[p * ld + q];
                    const double app = T[p * ld + p], aqq = T[q * ld + q];
                    if (fabs(apq) > atol && apq * apq > gtol * fabs(aqq - app)) {
                        const double tau = (aqq - app) / (2.0 * apq);
                        // a correctly rounded reciprocal is 1.0 / x, in half the time
                        const double r = __drcp_rn(fabs(tau) + hypot(1.0, tau)), t = tau >= 0.0 ? r : -r;
                        c = 1.0 / sqrt(1.0 + t * t);
                        s = t * c;
                        a = 1;
                    }
                }
                cs[k] = make_double2(c, s);
                act[k] = a;
                if (!fold) rb[((int64_t)sweep * (np - 1) + st) * m + k] = make_double2(c, s);
            }
            const int active = __syncthreads_count(a);
            if (active == 0) continue;
            nrot += active;
            // 2x2 blocks (P, Q) with P rotated; a block with both P and Q
            // rotated is handled once, by the smaller of the two
            for (int P = warp; P < m; P += warps) {
                if (!act[P]) continue;
                const double2 cp = cs[P];
                int pP, qP;
                rr_pair(st, P, np, pP, qP);
                for (int Q = lane; Q < m; Q += 32) {
                    if (act[Q] && Q < P) continue;
                    const double2 cq = cs[Q];
                    int pQ, qQ;
                    rr_pair(st, Q, np, pQ, qQ);
                    const double b11 = T[pP * ld + pQ], b12 = T[pP * ld + qQ];
                    const double b21 = T[qP * ld + pQ], b22 = T[qP * ld + qQ];
                    const double m11 = b11 * cq.x - b12 * cq.y, m12 = b11 * cq.y + b12 * cq.x;
                    const double m21 = b21 * cq.x - b22 * cq.y, m22 = b21 * cq.y + b22 * cq.x;
                    double n11 = cp.x * m11 - cp.y * m21, n12 = cp.x * m12 - cp.y * m22;
                    double n21 = cp.y * m11 + cp.x * m21, n22 = cp.y * m12 + cp.x * m22;
                    if (P == Q) {
                        n12 = 0.0;
                        n21 = 0.0;
                        T[pP * ld + pP] = n11;
                        T[pP * ld + qP] = n12;
                        T[qP * ld + pP] = n21;
                        T[qP * ld + qP] = n22;
                    } else {
                        T[pP * ld + pQ] = n11; T[pQ * ld + pP] = n11;
                        T[pP * ld + qQ] = n12; T[qQ * ld + pP] = n12;
                        T[qP * ld + pQ] = n21; T[pQ * ld + qP] = n21;
                        T[qP * ld + qQ] = n22; T[qQ * ld + qP] = n22;
                    }
                }
            }
            if (fold) rotate_V(st);
            __syncthreads();
        }
        total += nrot;
        if (nrot == 0) {
            sweep++;
            break;
        }
    }
    if (threadIdx.x == 0) {
        if (rot_count) atomicAdd(rot_count, total);
        if (sweep >= max_sweeps && nrot != 0) atomicAdd(status, 1);   // sweeps exhausted
    }

    // middle factor P of U+ = V P V^T (first-order in the remaining couplings)
    double *Pb = Pout + off;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = e / n, j = e % n;
        const double li = T[i * ld + i];
        double pv;
        if (raw) {
            pv = T[i * ld + j];   // the rotated matrix itself (its diagonal: the eigenvalues)
        } else if (i == j) {
            pv = fmax(li, 0.0);
        } else {
            const double lj = T[j * ld + j];
            const double pi = fmax(li, 0.0), pj = fmax(lj, 0.0);
            const double gam = (li != lj) ? (pi - pj) / (li - lj) : (li > 0.0 ? 1.0 : 0.0);
            pv = gam * T[i * ld + j];
        }
        Pb[e] = pv;
    }
    __syncthreads();

    if (!fold) {
        // replay the rotations on Vt; a step's are fetched during the one before
        load_V();
        const int steps = sweep * (np - 1), k = threadIdx.x;
        double2 r = k < m && steps > 0 ? rb[k] : make_double2(1.0, 0.0);
        for (int q = 0, st = 0; q < steps; q++, st = st + 1 == np - 1 ? 0 : st + 1) {
            if (k < m) {
                cs[k] = r;
                act[k] = r.y != 0.0;
            }
            const int active = __syncthreads_count(r.y != 0.0);
            if (k < m && q + 1 < steps) r = rb[(int64_t)(q + 1) * m + k];
            if (active) rotate_V(st);
            __syncthreads();
        }
    }
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = e / n, j = e % n;
        Vb[e] = V[i * ld + j];
    }
}

// Vt <- identity on every block (cold start of the warm path)
__global__ void identity_blocks_kernel(double *__restrict__ Vt, const int64_t *__restrict__ boff,
                                       const int *__restrict__ bdim) {
    const int n = bdim[blockIdx.x];
    const int64_t off = boff[blockIdx.x];
    for (int64_t e = threadIdx.x; e < (int64_t)n * n; e += blockDim.x)
        Vt[off + e] = (e / n == e % n) ? 1.0 : 0.0;
}

// H = (I - G) / 2 for the re-orthonormalisation Vt <- Vt + H Vt
__global__ void half_residual_kernel(const double *__restrict__ G, double *__restrict__ H,
                                     const int64_t *__restrict__ boff, const int *__restrict__ bdim) {
    const int n = bdim[blockIdx.x];
    const int64_t off = boff[blockIdx.x];
    for (int64_t e = threadIdx.x; e < (int64_t)n * n; e += blockDim.x)
        H[off + e] = 0.5 * (((e / n == e % n) ? 1.0 : 0.0) - G[off + e]);
}

cudaError_t raise_dynamic_smem(const void *func, int bytes) {
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, func);
    if (e == cudaSuccess && fa.maxDynamicSharedSizeBytes < bytes)
        e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e;
}

unsigned long long current_context_id() {
    // driver entry points through the runtime: no link-time libcuda dependency
    using GetCurrent = CUresult (*)(CUcontext *);
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static const std::pair<GetCurrent, GetId> fn = [] {
        void *a = nullptr, *b = nullptr;
        cudaDriverEntryPointQueryResult qa, qb;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &a, cudaEnableDefault, &qa) != cudaSuccess ||
            qa != cudaDriverEntryPointSuccess)
            a = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &b, cudaEnableDefault, &qb) != cudaSuccess ||
            qb != cudaDriverEntryPointSuccess)
            b = nullptr;
        return std::make_pair((GetCurrent)a, (GetId)b);
    }();
    if (!fn.first || !fn.second) return 0;
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (fn.first(&ctx) != CUDA_SUCCESS || !ctx) return 0;
    if (fn.second(ctx, &id) != CUDA_SUCCESS) return 0;
    return id;
}

}  // namespace v2b
