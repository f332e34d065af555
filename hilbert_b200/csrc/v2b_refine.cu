// Warm eigen-refinement of the per-block PSD projection (sm_100a).
//
// The projection needs U+ = V f(L) V^T with f(l) = max(l, 0).  The rows of
// Vt from the previous outer iteration nearly diagonalise the new block, so
// T = Vt U Vt^T = D + E with E small, and to first order
//     f(T) = Gamma o T,   Gamma_pq = (f(d_p) - f(d_q)) / (d_p - d_q)
// (Daleckii-Krein).  f is linear on each side of zero, so the first-order
// formula loses accuracy only through couplings between the two sides, and
// through couplings that blur the sign of a diagonal entry.  A pair (p, q) is
// accepted when
//     t_pq^2 <= gap_tol ||T||_F Delta_pq   or   |t_pq| <= abs_tol ||T||_F,
//     Delta_pq = |d_p - d_q|            (d_p, d_q of opposite sign)
//              = min(|d_p|, |d_q|)      (same sign: distance to zero)
// (the same tolerances as the Jacobi kernels' rotation test, with the gap
// replaced by the distance that governs f's second divided differences).
// A block whose pairs all pass takes P = Gamma o T directly.  Otherwise one
// pass refines Vt:
//   * non-separable failing pairs (|t_pq| > rho |d_p - d_q|) form a graph; its
//     connected components ("clusters", found on the host from the recorded
//     edges) are diagonalised exactly -- up to kRefineSmallCluster rows by
//     cluster_eig_kernel, larger ones gathered into compact matrices for the
//     selective Jacobi kernels with the gap test off -- and the rotation G
//     (identity outside the clusters) is applied as T <- G T G^T, Vt <- G Vt
//     with gathered GEMM tiles;
//   * every remaining separable failing pair takes one Newton step of the
//     eigenvector equation, Vt <- (I - K) Vt with K_pq = t_pq / (d_q - d_p),
//     followed by one Newton-Schulz orthonormalisation
//     Vt <- (3/2 I - 1/2 Vt Vt^T) Vt (GEMMs).  Accepted pairs take the step only
//     when it is tiny: inside a near-degenerate same-sign cluster t/(d_q - d_p)
//     is large and meaningless (f is linear there) and would only cost
//     orthogonality;
// and T is recomputed.  Blocks that still fail after kRefinePasses passes, or
// record more than kRefineEdgeCap non-separable pairs, fall back to the
// selective Jacobi kernels, restarted from the basis and T the call began with.
#include "v2b_kernels.cuh"
#include "v2b_refine.cuh"

#include <algorithm>

namespace v2b {

__device__ __forceinline__ double gamma_pq(double li, double lj) {
    const double pi = fmax(li, 0.0), pj = fmax(lj, 0.0);
    return (li != lj) ? (pi - pj) / (li - lj) : (li > 0.0 ? 1.0 : 0.0);
}

// CTA s of a block takes the row pairs (r, n-1-r), r in [s R, (s+1) R),
// R = ceil(ceil(n/2) / kNormSplit).
__device__ __forceinline__ void split_rows(int n, int s, int &r0, int &r1) {
    const int half = (n + 1) / 2, R = (half + kNormSplit - 1) / kNormSplit;
    r0 = min(half, s * R);
    r1 = min(half, (s + 1) * R);
}

// Frobenius norms of the symmetrised blocks, in kNormSplit partial sums per
// block (summed in a fixed order by the readers: the result is deterministic)
__global__ void __launch_bounds__(256)
    block_norm_kernel(const double *__restrict__ Us, const int64_t *__restrict__ boff,
                      const int *__restrict__ bdim, double *__restrict__ part) {
    const int blk = blockIdx.x, sidx = blockIdx.y, n = bdim[blk];
    __shared__ double red[32];
    int r0, r1;
    split_rows(n, sidx, r0, r1);
    const double *Ub = Us + boff[blk];
    double acc = 0.0;
    // the CTA's rows r0, n-1-r0, r0+1, ..., each in strides of the CTA; added
    // one by one, kBatch loads in flight
    constexpr int kBatch = 8;
    const int tid = threadIdx.x, rows = 2 * (r1 - r0) - (2 * r1 > n ? 1 : 0);   // the middle row once
    int u = 0, c = tid;
    while (u < rows && c < n) {
        double v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; k++) {
            const bool in = u < rows;   // else a load of no use, so that none waits for a branch
            const int r = r0 + (u >> 1), row = (u & 1) ? n - 1 - r : r;
            const double w = Ub[in ? (int64_t)row * n + c : 0];
            v[k] = in ? w : 0.0;
            const int next = c + (int)blockDim.x;
            u += next >= n;
            c = next >= n ? tid : next;
        }
#pragma unroll
        for (int k = 0; k < kBatch; k++) acc += v[k] * v[k];
    }
    acc = block_sum(acc, red);
    if (threadIdx.x == 0) part[blk * kNormSplit + sidx] = acc;
}

__device__ __forceinline__ double block_norm(const double *part, int blk) {
    double s = 0.0;
    for (int k = 0; k < kNormSplit; k++) s += part[blk * kNormSplit + k];
    return sqrt(s);
}

// Acceptance test, gridDim.y CTAs per block: the pairs of 32 x 32 tiles (I, J),
// (J, I), read along rows and turned in shared memory.  Failing pairs are
// counted and non-separable ones recorded as edges; the last CTA of a block to
// finish sets its state (done -> done_stamp = stamp, for write_p_kernel).
// (20e,20o), all blocks: 24 us; with columns read from memory by 16 CTAs a
// block 63.
__global__ void __launch_bounds__(kRefineThreads)
    refine_classify_kernel(const double *__restrict__ T, const int64_t *__restrict__ boff,
                           const int *__restrict__ bdim, int *__restrict__ bstate,
                           const unsigned long long *__restrict__ orth, const double *__restrict__ part,
                           double gap_tol, double abs_tol, double *__restrict__ bnorm,
                           int *__restrict__ counts, int *__restrict__ done_stamp, int stamp,
                           int *h_state, int *h_nbad, int *h_nedge, int2 *h_edges) {
    const int blk = blockIdx.x, sidx = blockIdx.y;
    const int st_in = bstate[blk];
    if (st_in != kStWork && st_in != kStBlockJacobi) return;   // uniform over the CTA
    const int n = bdim[blk];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
    int *cnt = counts + 3 * blk;   // [0] failing pairs, [1] edges, [2] finished CTAs
    __shared__ int s_last;
    __shared__ double up[32][33], lo[32][33], dg[2][32];   // T[I, J], T[J, I], their diagonals
    const int64_t off = boff[blk];
    const double *Tb = T + off;
    const double nrm = block_norm(part, blk);
    const double atol = abs_tol * nrm, gtol = gap_tol * nrm;
    int bad = 0;
    int2 *eb = h_edges + (int64_t)blk * kRefineEdgeCap;
    const int nt = (n + 31) / 32, npairs = nt * (nt + 1) / 2;
    for (int t = sidx; t < npairs; t += gridDim.y) {
        int I = 0, J = t;
        while (J >= nt - I) J -= nt - I++;
        J += I;
        const int i0 = 32 * I, j0 = 32 * J;
        __syncthreads();
        for (int r = warp; r < 32; r += nwarp) {
            up[r][lane] = i0 + r < n && j0 + lane < n ? Tb[(int64_t)(i0 + r) * n + j0 + lane] : 0.0;
            lo[r][lane] = j0 + r < n && i0 + lane < n ? Tb[(int64_t)(j0 + r) * n + i0 + lane] : 0.0;
        }
        if (warp < 2) {
            const int i = (warp ? j0 : i0) + lane;
            dg[warp][lane] = i < n ? Tb[(int64_t)i * n + i] : 0.0;
        }
        __syncthreads();
        for (int r = warp; r < 32; r += nwarp) {
            const int i = i0 + r, j = j0 + lane;
            if (j <= i || j >= n) continue;   // i < j < n
            const double t = 0.5 * (up[r][lane] + lo[lane][r]);
            const double at = fabs(t);
            if (at <= atol) continue;
            const double di = dg[0][r], dj = dg[1][lane];
            const double g = fabs(di - dj);
            const bool cross = (di >= 0.0) != (dj >= 0.0);
            const double delta = cross ? g : fmin(fabs(di), fabs(dj));
            if (t * t > gtol * delta) {
                bad++;
                if (at > kRefineRho * g) {
                    const int e = atomicAdd(cnt + 1, 1);
                    if (e < kRefineEdgeCap) eb[e] = make_int2(i, j);
                }
            }
        }
    }
    __syncwarp();
    bad = __reduce_add_sync(0xffffffffu, bad);
    if (lane == 0 && bad) atomicAdd(cnt, bad);
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = (atomicAdd(cnt + 2, 1) == (int)gridDim.y - 1);
    __syncthreads();
    if (!s_last) return;
    if (tid == 0) {
        __threadfence();
        const int nbad = atomicAdd(cnt, 0), ne = atomicAdd(cnt + 1, 0);
        const bool done = nbad == 0 && __longlong_as_double((long long)orth[blk]) <= kRefineOrthDone;
        const int st = done ? kStDone : st_in;
        if (done) done_stamp[blk] = stamp;
        bstate[blk] = st;
        bnorm[blk] = nrm;
        h_state[blk] = st;
        h_nbad[blk] = nbad;
        h_nedge[blk] = ne;
        cnt[0] = cnt[1] = cnt[2] = 0;   // ready for the next launch
    }
}

// P = Gamma o T on the tiles of the blocks accepted by the classify launch
// with this stamp
__global__ void __launch_bounds__(256)
    write_p_kernel(const double *__restrict__ T, double *__restrict__ P,
                   const int4 *__restrict__ tiles, const int64_t *__restrict__ boff,
                   const int *__restrict__ bdim, const int *__restrict__ done_stamp, int stamp) {
    const int4 t = tiles[blockIdx.x];
    if (done_stamp[t.x] != stamp) return;
    const int n = bdim[t.x];
    const int64_t off = boff[t.x];
    const double *Tb = T + off;
    double *Pb = P + off;
    for (int e = threadIdx.x; e < 64 * 64; e += blockDim.x) {
        const int i = t.y * 64 + e / 64, j = t.z * 64 + e % 64;
        if (i >= n || j >= n) continue;
        const double di = Tb[(int64_t)i * n + i];
        double v;
        if (i == j) {
            v = fmax(di, 0.0);
        } else {
            const double dj = Tb[(int64_t)j * n + j];
            v = gamma_pq(di, dj) * 0.5 * (Tb[(int64_t)i * n + j] + Tb[(int64_t)j * n + i]);
        }
        Pb[(int64_t)i * n + j] = v;
    }
}

// ---------------------------------------------------------------- clusters
// Cyclic Jacobi on one cluster (k <= kRefineSmallCluster), A and the
// eigenvector rows Q in shared memory.  A step takes the m = kp / 2 disjoint
// round-robin pairs (sym.schur2 rotations), each 2 x 2 block (rows of pair P,
// columns of pair Q2) two-sidedly, and the rows p, q of Q.
//
// A step is a chain: the rotations' divisions and roots (600 cycles alone),
// then the update, which is bound by shared memory (every element of A and Q
// is read and written).  So the chain runs beside the update: a warp of its
// own forms the three elements that each next pair needs from the blocks as
// they stand before the update, then the next rotations, while the others
// write A and update Q; they wait only until it has read.  And the columns of
// Q are cut over `slices` CTAs, each of which repeats the whole of A (the same
// bits): no exchange, and Q's traffic, half of a step's, is divided.  A
// 64-row job, two sweeps: 216 us with the rotations and the updates in turn
// and one CTA a job, 137 us so.
__device__ __forceinline__ void bar_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
struct RotBlock {
    double n11, n12, n21, n22;
};
// the 2 x 2 block b of pairs (P, Q2) after both rotations; same: P == Q2, the
// pair's own coupling is annihilated
__device__ __forceinline__ RotBlock rotate_block(double b11, double b12, double b21, double b22, double2 cp,
                                                 double2 cq, bool same) {
    const double m11 = b11 * cq.x - b12 * cq.y, m12 = b11 * cq.y + b12 * cq.x;
    const double m21 = b21 * cq.x - b22 * cq.y, m22 = b21 * cq.y + b22 * cq.x;
    RotBlock r;
    r.n11 = cp.x * m11 - cp.y * m21;
    r.n12 = cp.x * m12 - cp.y * m22;
    r.n21 = cp.y * m11 + cp.x * m21;
    r.n22 = cp.y * m12 + cp.x * m22;
    if (same) r.n12 = r.n21 = 0.0;
    return r;
}
// rr_pair without divisions, and its inverse: the pair that holds index j
__device__ __forceinline__ void rr_pair_fast(int s, int k, int m1, int &p, int &q) {
    int a = s + k, b = s - k;
    a = a >= m1 ? a - m1 : a;
    b = b < 0 ? b + m1 : b;
    a = k == 0 ? m1 : a;
    p = min(a, b);
    q = max(a, b);
}
// what the rotating warp needs of step st for pair `lane` of the next step
// (p, q): each index's partner and pair in step st
__device__ __forceinline__ uint2 next_pair_entry(int st, int nx, int lane, int m1) {
    auto pair_of = [&](int j) {
        if (j == m1 || j == st) return 0;
        const int d = j > st ? j - st : j - st + m1;
        return min(d, m1 - d);
    };
    int p, q, a, b, c, d;
    rr_pair_fast(nx, lane, m1, p, q);
    const int Pp = pair_of(p), Pq = pair_of(q);
    rr_pair_fast(st, Pp, m1, a, b);
    rr_pair_fast(st, Pq, m1, c, d);
    return make_uint2((unsigned)(p | (a + b - p) << 8 | Pp << 16), (unsigned)(q | (c + d - q) << 8 | Pq << 16));
}

// NT threads update, a warp per pair row P and a lane per pair column; one more
// warp rotates.  NT = 128: at most 32 rows (16 pairs).
template <int NT>
__global__ void __launch_bounds__(NT + 32)
    cluster_eig_kernel(const double *__restrict__ T, const int64_t *__restrict__ boff,
                       const int *__restrict__ bdim, const ClusterJob *__restrict__ jobs,
                       const int *__restrict__ mem, double *__restrict__ Qt,
                       double *__restrict__ lam, const int *__restrict__ only, int max_sweeps, int slices) {
    const ClusterJob jb = jobs[blockIdx.x / slices];
    if (only && !only[jb.blk]) return;   // uniform over the CTA
    constexpr int KM = kRefineSmallCluster, WARPS = NT / 32, PASSES = 2 * (NT > 128 ? 16 : 8) / WARPS;
    const int k = jb.k, n = bdim[jb.blk];
    const int kp = k + (k & 1), ld = kp + 1, m = kp / 2, nst = kp - 1;
    // this CTA's columns of Q
    const int cw = (kp + slices - 1) / slices, c0 = (int)(blockIdx.x % slices) * cw, c1 = min(kp, c0 + cw);
    if (c0 >= c1 && c0 > 0) return;   // uniform over the CTA
    const int *C = mem + jb.moff;
    const double *Tb = T + boff[jb.blk];
    extern __shared__ double sm[];
    double *A = sm;              // kp x ld
    double *Q = A + kp * ld;     // kp x cw, rows = eigenvectors
    uint2 *next = (uint2 *)(Q + kp * cw);   // nst x m
    __shared__ double2 cs[3][KM / 2];   // the step before, this one, the next
    __shared__ double red[32];
    __shared__ double s_thr;
    __shared__ int s_any[2];
    const int tid = threadIdx.x;
    double fro = 0.0;
    for (int e = tid; e < kp * kp; e += blockDim.x) {
        const int i = e / kp, j = e % kp;
        double v = 0.0;
        if (i < k && j < k) {
            const int64_t a = C[i], b = C[j];
            v = 0.5 * (Tb[a * n + b] + Tb[b * n + a]);
        }
        A[i * ld + j] = v;
        if (j >= c0 && j < c1) Q[i * cw + j - c0] = (i == j) ? 1.0 : 0.0;
        fro += v * v;
    }
    for (int e = tid; e < nst * m; e += blockDim.x) {
        const int st = e / m;
        next[e] = next_pair_entry(st, st + 1 < nst ? st + 1 : 0, e % m, nst);
    }
    fro = block_sum(fro, red);
    // rotate down to 1e-14 of the cluster's norm: below the acceptance test's
    // floor (1e-14 of the block's norm) and above the rounding noise the
    // rotations themselves leave, so the sweeps end
    if (tid == 0) s_thr = 1e-14 * sqrt(fro) + 1e-300;
    __syncthreads();
    const double thr = s_thr;
    const int m1 = nst;
    // the rotation of the pair with elements app, aqq, apq (q < k: not padding)
    auto rotation = [&](int q, double app, double aqq, double apq) {
        double c = 1.0, s = 0.0;
        if (q < k && fabs(apq) > thr) {
            const double tau = (aqq - app) / (2.0 * apq);
            // a correctly rounded reciprocal is 1.0 / x, in half the time
            const double r = __drcp_rn(fabs(tau) + hypot(1.0, tau)), t = tau >= 0.0 ? r : -r;
            c = 1.0 / sqrt(1.0 + t * t);
            s = t * c;
        }
        return make_double2(c, s);
    };
    if (tid >= NT) {   // the rotating warp; its lanes keep this step's rotations
        const int lane = tid - NT;
        double2 mine = make_double2(1.0, 0.0);
        bool any = false;   // a pair was rotated in this sweep
        if (lane < m) {
            int p, q;
            rr_pair_fast(0, lane, m1, p, q);
            mine = rotation(q, A[p * ld + p], A[q * ld + q], A[p * ld + q]);
            cs[0][lane] = mine;
            any = mine.y != 0.0;
        }
        __syncthreads();
        int cur = 0;
        uint2 e = lane < m ? next[lane] : make_uint2(0u, 0u);
        for (int sweep = 0; sweep < max_sweeps; sweep++) {
            for (int st = 0; st < nst; st++) {
                const int p = e.x & 255, p2 = (e.x >> 8) & 255, Pp = e.x >> 16;
                const int q = e.y & 255, q2 = (e.y >> 8) & 255, Pq = e.y >> 16;
                const double2 cp = make_double2(__shfl_sync(0xffffffffu, mine.x, Pp), __shfl_sync(0xffffffffu, mine.y, Pp));
                const double2 cq = make_double2(__shfl_sync(0xffffffffu, mine.x, Pq), __shfl_sync(0xffffffffu, mine.y, Pq));
                const int pp = min(p, p2), pq = max(p, p2), qp = min(q, q2), qq = max(q, q2);
                // rows and columns (pp, pq) x (pp, pq), (qp, qq) x (qp, qq) and
                // (pp, pq) x (qp, qq) of A as they stand
                const double a11 = A[pp * ld + pp], a12 = A[pp * ld + pq], a21 = A[pq * ld + pp], a22 = A[pq * ld + pq];
                const double b11 = A[qp * ld + qp], b12 = A[qp * ld + qq], b21 = A[qq * ld + qp], b22 = A[qq * ld + qq];
                const double x11 = A[pp * ld + qp], x12 = A[pp * ld + qq], x21 = A[pq * ld + qp], x22 = A[pq * ld + qq];
                const RotBlock ra = rotate_block(a11, a12, a21, a22, cp, cp, true);
                const RotBlock rb = rotate_block(b11, b12, b21, b22, cq, cq, true);
                const RotBlock rx = rotate_block(x11, x12, x21, x22, cp, cq, Pp == Pq && cp.y != 0.0);
                const double app = p == pp ? ra.n11 : ra.n22, aqq = q == qp ? rb.n11 : rb.n22;
                const double lo = q == qp ? rx.n11 : rx.n12, hi = q == qp ? rx.n21 : rx.n22;
                const double apq = p == pp ? lo : hi;
                bar_arrive(1, NT + 32);   // this step's A has been read
                // the next sweep's rotations begin in this sweep's last step
                if (st + 1 == nst) {
                    const int rotated = __any_sync(0xffffffffu, any);
                    if (lane == 0) s_any[sweep & 1] = rotated;
                    any = false;
                }
                if (lane < m) {
                    mine = rotation(q, app, aqq, apq);
                    cs[cur == 2 ? 0 : cur + 1][lane] = mine;
                    any = any || mine.y != 0.0;
                    e = next[(st + 1 < nst ? st + 1 : 0) * m + lane];
                }
                __syncwarp();
                cur = cur == 2 ? 0 : cur + 1;
                __syncthreads();
            }
            if (!s_any[sweep & 1]) break;
        }
    } else {
        __syncthreads();
        const int warp = tid >> 5, lane = tid & 31;
        const bool col = lane < m;   // this lane has a pair column
        // Q <- G Q of step st, rotations cs[c], this CTA's columns: the warp's
        // pair rows side by side over its lanes
        auto update_Q = [&](int st, int c) {
            for (int f = lane; f < PASSES * cw; f += 32) {
                const int i = f / cw, jc = f - i * cw, P = warp + i * WARPS;
                if (P >= m || jc >= c1 - c0) continue;
                const double2 g = cs[c][P];
                if (g.y == 0.0) continue;
                int p, q;
                rr_pair_fast(st, P, m1, p, q);
                const double qp = Q[p * cw + jc], qq = Q[q * cw + jc];
                Q[p * cw + jc] = g.x * qp - g.y * qq;
                Q[q * cw + jc] = g.y * qp + g.x * qq;
            }
        };
        int cur = 0, last = -1;   // last: the step whose rotations Q still lacks
        for (int sweep = 0; sweep < max_sweeps; sweep++) {
            for (int st = 0; st < nst; st++) {
                // Q first: the rotating warp's reads of A go ahead of these warps'
                if (last >= 0) update_Q(last, cur == 0 ? 2 : cur - 1);
                // A <- G A G^T on the 2 x 2 blocks (P, lane), held until all are
                // read.  Without a rotation a block comes out as it went in.
                RotBlock r[PASSES];
                int pP[PASSES], qP[PASSES], pQ, qQ;
                double2 cp[PASSES];
                const double2 cq = cs[cur][col ? lane : 0];
                rr_pair_fast(st, col ? lane : 0, m1, pQ, qQ);
#pragma unroll
                for (int i = 0; i < PASSES; i++) {
                    const int P = min(warp + i * WARPS, m - 1);
                    cp[i] = cs[cur][P];
                    rr_pair_fast(st, P, m1, pP[i], qP[i]);
                }
                double a[PASSES][4];
#pragma unroll
                for (int i = 0; i < PASSES; i++) {
                    a[i][0] = A[pP[i] * ld + pQ];
                    a[i][1] = A[pP[i] * ld + qQ];
                    a[i][2] = A[qP[i] * ld + pQ];
                    a[i][3] = A[qP[i] * ld + qQ];
                }
#pragma unroll
                for (int i = 0; i < PASSES; i++)
                    r[i] = rotate_block(a[i][0], a[i][1], a[i][2], a[i][3], cp[i], cq,
                                        lane == warp + i * WARPS && cq.y != 0.0);
                bar_sync(1, NT + 32);
#pragma unroll
                for (int i = 0; i < PASSES; i++)
                    if (col && warp + i * WARPS < m) {
                        A[pP[i] * ld + pQ] = r[i].n11;
                        A[pP[i] * ld + qQ] = r[i].n12;
                        A[qP[i] * ld + pQ] = r[i].n21;
                        A[qP[i] * ld + qQ] = r[i].n22;
                    }
                last = st;
                cur = cur == 2 ? 0 : cur + 1;
                __syncthreads();
            }
            if (!s_any[sweep & 1]) break;
        }
        if (last >= 0) update_Q(last, cur == 0 ? 2 : cur - 1);
    }
    __syncthreads();
    double *Qo = Qt + jb.qoff;
    for (int e = tid; e < k * cw; e += blockDim.x) {
        const int i = e / cw, j = c0 + e % cw;
        if (j < min(k, c1)) Qo[i * k + j] = Q[i * cw + e % cw];
    }
    if (c0 == 0)
        for (int i = tid; i < k; i += blockDim.x) lam[jb.moff + i] = A[i * ld + i];
}

// A, Q and the table of next pairs (one 8-byte entry per pair and step)
static size_t cluster_eig_smem(int kp, int cw) {
    return sizeof(double) * ((size_t)kp * (kp + 1) + (size_t)kp * cw + (size_t)(kp - 1) * (kp / 2));
}

cudaError_t launch_cluster_eig(int njobs, int kmax, int sms, cudaStream_t s, const double *T, const int64_t *boff,
                               const int *bdim, const ClusterJob *jobs, const int *mem, double *Qt, double *lam,
                               const int *only, int max_sweeps) {
    if (njobs <= 0) return cudaSuccess;
    const int kp = kmax + (kmax & 1);
    // columns of Q over as many CTAs as the SMs hold at once, at least 16 each
    const int slices = std::max(1, std::min({4, kp / 16, sms / njobs}));
    const size_t smem = cluster_eig_smem(kp, (kp + slices - 1) / slices);
    if (kp > 32)
        cluster_eig_kernel<512><<<njobs * slices, 512 + 32, smem, s>>>(T, boff, bdim, jobs, mem, Qt, lam, only,
                                                                      max_sweeps, slices);
    else
        cluster_eig_kernel<128><<<njobs * slices, 128 + 32, smem, s>>>(T, boff, bdim, jobs, mem, Qt, lam, only,
                                                                      max_sweeps, slices);
    return cudaGetLastError();
}

cudaError_t prepare_cluster_eig() {
    const int kc = kRefineSmallCluster;
    const int smem = (int)cluster_eig_smem(kc, kc);
    cudaError_t e = raise_dynamic_smem((const void *)cluster_eig_kernel<512>, smem);
    return e == cudaSuccess ? raise_dynamic_smem((const void *)cluster_eig_kernel<128>, smem) : e;
}

// One block-Jacobi step applied in place.  The step's jobs partition each
// block's rows, so T splits into job tiles T[C_I, C_J] that only their own
// CTA reads and writes:  tile kind 0 (I, J):  T[C_I, C_J] <- Qt_I T[C_I, C_J] Qt_J^T;
// kind 1 (I, t):  Vt[C_I, 64 t .. 64 t + 64) <- Qt_I Vt[C_I, ...].
//
// 64 x 64 x 64 products on FP64 tensor cores (m8n8k4; its four products
// accumulate in ascending k with one rounding each, bit for bit an FMA chain),
// eight warps of 32 x 16 each: 8 fragment loads feed 8 MMAs, where FMAs from
// shared memory were bound by their operand loads (45 us a launch at 200 rows
// then, 25 now with cold caches; 4 us of it are the MMAs of one tile).
constexpr int kBjLd = kRefineSmallCluster + 4;   // rows 4 doubles apart mod 16: fragments free of conflicts

// c += op(X) Y over K = 64 (zero-padded): rows wm.., columns wn..; X row-major
// 64 x 64; Y row-major (k x n), or with YT its transpose (n x k)
template <bool YT>
__device__ __forceinline__ void bj_mma(const double *X, const double *Y, int wm, int wn, int lane, int kmax,
                                       double (&c)[4][2][2]) {
    const int fr = lane >> 2, fk = lane & 3;
    for (int k = 0; k < kmax; k += 4) {
        double x[4], y[2];
#pragma unroll
        for (int i = 0; i < 4; i++) x[i] = X[(wm + 8 * i + fr) * kBjLd + k + fk];
#pragma unroll
        for (int j = 0; j < 2; j++)
            y[j] = YT ? Y[(wn + 8 * j + fr) * kBjLd + k + fk] : Y[(k + fk) * kBjLd + wn + 8 * j + fr];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 2; j++)
                asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                             : "+d"(c[i][j][0]), "+d"(c[i][j][1])
                             : "d"(x[i]), "d"(y[j]));
    }
}

__global__ void __launch_bounds__(256)
    bj_apply_kernel(double *__restrict__ T, double *__restrict__ Vt, const int64_t *__restrict__ boff,
                    const int *__restrict__ bdim, const ClusterJob *__restrict__ jobs,
                    const int *__restrict__ mem, const double *__restrict__ Qt,
                    const int4 *__restrict__ tiles, const int *__restrict__ only) {
    const int4 tl = tiles[blockIdx.x];
    const ClusterJob jI = jobs[tl.x];
    if (only && !only[jI.blk]) return;   // uniform over the CTA
    const int n = bdim[jI.blk];
    const int64_t off = boff[jI.blk];
    constexpr int KM = kRefineSmallCluster, SZ = KM * kBjLd;
    extern __shared__ double sm[];
    double *sQ = sm;              // Qt_I, zero past its kI rows and columns
    double *sX = sm + SZ;         // the tile, then Qt_I x tile
    double *sR = sm + 2 * SZ;     // Qt_J (kind 0)
    __shared__ int rI[KM], rJ[KM];   // global rows; columns of kind 1
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp >> 2) * 32, wn = (warp & 3) * 16;
    const int kI = jI.k;
    const bool two = tl.z == 0;
    int kJ = 64;
    if (tid < KM) rI[tid] = tid < kI ? mem[jI.moff + tid] : 0;
    ClusterJob jJ = jI;
    if (two) {
        jJ = jobs[tl.y];
        kJ = jJ.k;
        if (tid < KM) rJ[tid] = tid < kJ ? mem[jJ.moff + tid] : 0;
    } else {
        const int c0 = tl.y * 64;
        kJ = min(64, n - c0);
        if (tid < KM) rJ[tid] = c0 + min(tid, kJ - 1);
    }
    __syncthreads();
    double *G = (two ? T : Vt) + off;
#pragma unroll 8
    for (int e = tid; e < KM * KM; e += 256) {
        const int i = e >> 6, j = e & 63;
        sQ[i * kBjLd + j] = i < kI && j < kI ? Qt[jI.qoff + i * kI + j] : 0.0;
        sX[i * kBjLd + j] = i < kI && j < kJ ? G[(int64_t)rI[i] * n + rJ[j]] : 0.0;
        if (two) sR[i * kBjLd + j] = i < kJ && j < kJ ? Qt[jJ.qoff + i * kJ + j] : 0.0;
    }
    __syncthreads();
    const int fr = lane >> 2, fk = lane & 3;
    double c[4][2][2] = {};
    bj_mma<false>(sQ, sX, wm, wn, lane, (kI + 3) & ~3, c);   // Y = Qt_I X
    if (two) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    sX[(wm + 8 * i + fr) * kBjLd + wn + 8 * j + 2 * fk + h] = c[i][j][h];
                    c[i][j][h] = 0.0;
                }
        __syncthreads();
        bj_mma<true>(sX, sR, wm, wn, lane, (kJ + 3) & ~3, c);   // Z = Y Qt_J^T
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = wm + 8 * i + fr;
        if (r >= kI) continue;
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int q = wn + 8 * j + 2 * fk + h;
                if (q < kJ) G[(int64_t)rI[r] * n + rJ[q]] = c[i][j][h];
            }
    }
}

// Gathered GEMM tiles of the cluster transform G (identity outside the
// clusters, Qt on each cluster): tile (job, ti, tc) of
//     W[C_i, c]   = sum_l Qt[i][l] T[C_l, c],   Vt2[C_i, c] = sum_l Qt[i][l] Vt[C_l, c]
// for i in [32 ti, 32 ti + 32), c in [64 tc, 64 tc + 64).
__global__ void __launch_bounds__(256)
    cluster_rows_kernel(const double *__restrict__ T, const double *__restrict__ Vt,
                        double *__restrict__ W, double *__restrict__ Vt2,
                        const int64_t *__restrict__ boff, const int *__restrict__ bdim,
                        const ClusterJob *__restrict__ jobs, const int *__restrict__ mem,
                        const double *__restrict__ Qt, const int4 *__restrict__ ctiles,
                        const int *__restrict__ only) {
    const int4 ct = ctiles[blockIdx.x];
    const ClusterJob jb = jobs[ct.x];
    if (only && !only[jb.blk]) return;
    const int k = jb.k, n = bdim[jb.blk];
    const int i0 = ct.y * 32, c0 = ct.z * 64;
    const int64_t off = boff[jb.blk];
    const int *C = mem + jb.moff;
    const double *Q = Qt + jb.qoff;
    __shared__ double sQ[32][17];
    __shared__ double sT[16][65], sV[16][65];
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    double aT[2][4] = {}, aV[2][4] = {};
    for (int l0 = 0; l0 < k; l0 += 16) {
        for (int e = tid; e < 32 * 16; e += 256) {
            const int ii = e >> 4, ll = e & 15;
            const int i = i0 + ii, l = l0 + ll;
            sQ[ii][ll] = (i < k && l < k) ? Q[(int64_t)i * k + l] : 0.0;
        }
        for (int e = tid; e < 16 * 64; e += 256) {
            const int ll = e >> 6, cc = e & 63;
            const int l = l0 + ll, c = c0 + cc;
            double vt = 0.0, vv = 0.0;
            if (l < k && c < n) {
                const int64_t idx = off + (int64_t)C[l] * n + c;
                vt = T[idx];
                vv = Vt[idx];
            }
            sT[ll][cc] = vt;
            sV[ll][cc] = vv;
        }
        __syncthreads();
#pragma unroll
        for (int ll = 0; ll < 16; ll++) {
            const double q0 = sQ[ty * 2][ll], q1 = sQ[ty * 2 + 1][ll];
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
                const double bt = sT[ll][tx * 4 + jj], bv = sV[ll][tx * 4 + jj];
                aT[0][jj] = fma(q0, bt, aT[0][jj]);
                aT[1][jj] = fma(q1, bt, aT[1][jj]);
                aV[0][jj] = fma(q0, bv, aV[0][jj]);
                aV[1][jj] = fma(q1, bv, aV[1][jj]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int i = i0 + ty * 2 + r;
        if (i >= k) continue;
#pragma unroll
        for (int jj = 0; jj < 4; jj++) {
            const int c = c0 + tx * 4 + jj;
            if (c >= n) continue;
            const int64_t idx = off + (int64_t)C[i] * n + c;
            W[idx] = aT[r][jj];
            Vt2[idx] = aV[r][jj];
        }
    }
}

// tile (job, ta, ti): P[a, C_i] = sum_l R(a)[C_l] Qt[i][l] for a in [64 ta, 64 ta + 64),
// i in [32 ti, 32 ti + 32), with R(a) = W[a, :] on cluster rows (already
// rotated by their own cluster) and T[a, :] elsewhere.  The cluster's own
// block comes out as Qt T[C, C] Qt^T: diagonal when the cluster solve was
// exact, and still the rotated block when its sweeps were capped.  P is free
// scratch for blocks in refinement.
__global__ void __launch_bounds__(256)
    cluster_cols_kernel(const double *__restrict__ T, const double *__restrict__ W,
                        double *__restrict__ P, const int64_t *__restrict__ boff,
                        const int *__restrict__ bdim, const ClusterJob *__restrict__ jobs,
                        const int *__restrict__ mem, const int *__restrict__ rowclus,
                        const int *__restrict__ rowbase, const double *__restrict__ Qt,
                        const double *__restrict__ lam, const int4 *__restrict__ ctiles,
                        const int *__restrict__ only) {
    const int4 ct = ctiles[blockIdx.x];
    const int jid = ct.x;
    const ClusterJob jb = jobs[jid];
    if (only && !only[jb.blk]) return;
    const int k = jb.k, n = bdim[jb.blk];
    const int a0 = ct.y * 64, i0 = ct.z * 32;
    const int64_t off = boff[jb.blk];
    const int *C = mem + jb.moff;
    const int *rc = rowclus + rowbase[jb.blk];
    const double *Q = Qt + jb.qoff;
    __shared__ double sR[64][17];
    __shared__ double sQ[32][17];
    const int tid = threadIdx.x, ta = tid >> 3, ti = tid & 7;
    double acc[2][4] = {};
    for (int l0 = 0; l0 < k; l0 += 16) {
        for (int e = tid; e < 64 * 16; e += 256) {
            const int aa = e >> 4, ll = e & 15;
            const int a = a0 + aa, l = l0 + ll;
            double v = 0.0;
            if (a < n && l < k) v = (rc[a] >= 0 ? W : T)[off + (int64_t)a * n + C[l]];
            sR[aa][ll] = v;
        }
        for (int e = tid; e < 32 * 16; e += 256) {
            const int ii = e >> 4, ll = e & 15;
            const int i = i0 + ii, l = l0 + ll;
            sQ[ii][ll] = (i < k && l < k) ? Q[(int64_t)i * k + l] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int ll = 0; ll < 16; ll++) {
            const double r0 = sR[ta * 2][ll], r1 = sR[ta * 2 + 1][ll];
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
                const double q = sQ[ti * 4 + jj][ll];
                acc[0][jj] = fma(r0, q, acc[0][jj]);
                acc[1][jj] = fma(r1, q, acc[1][jj]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int a = a0 + ta * 2 + r;
        if (a >= n) continue;
#pragma unroll
        for (int jj = 0; jj < 4; jj++) {
            const int i = i0 + ti * 4 + jj;
            if (i >= k) continue;
            P[off + (int64_t)a * n + C[i]] = acc[r][jj];
        }
    }
}

// tile (job, t): T[a, C_i] = P[a, C_i] for rows a in [64 t, 64 t + 64), and
// for columns b in that range outside every cluster T[C_i, b] = W[C_i, b];
// Vt[C_i, b] = Vt2[C_i, b] for every b in the range.
__global__ void __launch_bounds__(256)
    cluster_commit_kernel(double *__restrict__ T, const double *__restrict__ W,
                          const double *__restrict__ P, double *__restrict__ Vt,
                          const double *__restrict__ Vt2, const int64_t *__restrict__ boff,
                          const int *__restrict__ bdim, const ClusterJob *__restrict__ jobs,
                          const int *__restrict__ mem, const int *__restrict__ rowclus,
                          const int *__restrict__ rowbase, const int4 *__restrict__ ctiles,
                          const int *__restrict__ only) {
    const int4 ct = ctiles[blockIdx.x];
    const ClusterJob jb = jobs[ct.x];
    if (only && !only[jb.blk]) return;
    const int k = jb.k, n = bdim[jb.blk];
    const int t0 = ct.y * 64;
    const int64_t off = boff[jb.blk];
    const int *C = mem + jb.moff;
    const int *rc = rowclus + rowbase[jb.blk];
    for (int e = threadIdx.x; e < 64 * k; e += blockDim.x) {
        const int i = e / 64, x = t0 + e % 64;
        if (x >= n) continue;
        const int64_t col = off + (int64_t)x * n + C[i];   // (row x, cluster column C_i)
        T[col] = P[col];
        const int64_t row = off + (int64_t)C[i] * n + x;   // (cluster row C_i, column x)
        if (rc[x] < 0) T[row] = W[row];
        Vt[row] = Vt2[row];
    }
}

// Tc = sym(T[C, C]) and Vc = I in compact k x k storage at qoff, for clusters
// diagonalised by the Jacobi kernels (grid: jobs x 16, grid-stride inside)
__global__ void __launch_bounds__(256)
    cluster_gather_kernel(const double *__restrict__ T, const int64_t *__restrict__ boff,
                          const int *__restrict__ bdim, const ClusterJob *__restrict__ jobs,
                          const int *__restrict__ mem, const int *__restrict__ jlist,
                          double *__restrict__ Tc, double *__restrict__ Vc) {
    const ClusterJob jb = jobs[jlist[blockIdx.x]];
    const int k = jb.k, n = bdim[jb.blk];
    const int *C = mem + jb.moff;
    const double *Tb = T + boff[jb.blk];
    const int64_t kk = (int64_t)k * k;
    for (int64_t e = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; e < kk;
         e += (int64_t)gridDim.y * blockDim.x) {
        const int i = (int)(e / k), j = (int)(e % k);
        const int64_t a = C[i], b = C[j];
        Tc[jb.qoff + e] = 0.5 * (Tb[a * n + b] + Tb[b * n + a]);
        Vc[jb.qoff + e] = (i == j) ? 1.0 : 0.0;
    }
}

// lam[moff + i] = D[qoff + i k + i]: the eigenvalues left on the diagonal of
// the rotated compact matrix D by the Jacobi kernels
__global__ void cluster_lam_kernel(const ClusterJob *__restrict__ jobs, const int *__restrict__ jlist,
                                   int njobs, const double *__restrict__ Dsmall,
                                   const double *__restrict__ Dbig, int big_from,
                                   double *__restrict__ lam) {
    for (int q = blockIdx.x; q < njobs; q += gridDim.x) {
        const ClusterJob jb = jobs[jlist[q]];
        const double *D = (q >= big_from ? Dbig : Dsmall) + jb.qoff;
        for (int i = threadIdx.x; i < jb.k; i += blockDim.x) lam[jb.moff + i] = D[(int64_t)i * jb.k + i];
    }
}

// ---------------------------------------------------------------- Newton
__global__ void __launch_bounds__(256)
    newton_m_kernel(const double *__restrict__ T, double *__restrict__ M,
                    const int4 *__restrict__ tiles, const int64_t *__restrict__ boff,
                    const int *__restrict__ bdim, const int *__restrict__ bstate,
                    const double *__restrict__ bnorm, double gap_tol, double abs_tol) {
    const int4 t = tiles[blockIdx.x];
    if (bstate[t.x] != kStWork) return;
    const int n = bdim[t.x];
    const int64_t off = boff[t.x];
    const double *Tb = T + off;
    const double nrm = bnorm[t.x];
    const double atol = abs_tol * nrm, gtol = gap_tol * nrm;
    for (int e = threadIdx.x; e < 64 * 64; e += blockDim.x) {
        const int r = t.y * 64 + e / 64, c = t.z * 64 + e % 64;
        if (r >= n || c >= n) continue;
        double v;
        if (r == c) {
            v = 1.0;
        } else {
            const double tv = 0.5 * (Tb[(int64_t)r * n + c] + Tb[(int64_t)c * n + r]);
            const double dr = Tb[(int64_t)r * n + r], dc = Tb[(int64_t)c * n + c];
            const double g = dc - dr;
            v = 0.0;
            if (tv != 0.0 && fabs(tv) <= kRefineRho * fabs(g)) {
                const double k = tv / g;
                const bool cross = (dr >= 0.0) != (dc >= 0.0);
                const double delta = cross ? fabs(g) : fmin(fabs(dr), fabs(dc));
                const bool bad = fabs(tv) > atol && tv * tv > gtol * delta;
                if (bad || fabs(k) <= kRefineKappa) v = -k;
            }
        }
        M[off + (int64_t)r * n + c] = v;
    }
}

}  // namespace v2b
