#include "cg_tables.h"

#include <algorithm>
#include <stdexcept>

namespace v2b {

namespace {

constexpr uint32_t kNone = 0xffffffffu;

inline uint32_t code_of(uint32_t w) { return (w >> 27) & 15u; }
inline uint32_t length(const PackedOperator &op, int64_t r) { return op.row_ptr[r + 1] - op.row_ptr[r]; }

// positions and slice widths (off); the entries come later
void lay_out(const PackedOperator &op, CgSide &S) {
    S.off.assign(1, 0);
    std::vector<std::vector<uint32_t>> by_len(kCgLongRow + 1);
    std::vector<uint32_t> longs;
    for (int64_t w0 = 0; w0 < op.nrows; w0 += kCgSigma) {
        const int64_t w1 = std::min(op.nrows, w0 + kCgSigma);
        for (auto &v : by_len) v.clear();
        for (int64_t r = w0; r < w1; r++) {
            const uint32_t L = length(op, r);
            if (L <= kCgLongRow) by_len[L].push_back((uint32_t)r);
            else longs.push_back((uint32_t)r);
        }
        uint32_t lane = 0, width = 0;
        for (int L = (int)kCgLongRow; L >= 0; L--)
            for (const uint32_t r : by_len[L]) {
                if (lane == 0) width = (uint32_t)L;
                S.orig.push_back(r);
                S.len.push_back((uint8_t)L);
                if (++lane == 32) {
                    S.off.push_back(S.off.back() + 32u * width);
                    lane = 0;
                }
            }
        if (lane) {
            S.orig.insert(S.orig.end(), 32 - lane, kNone);
            S.len.insert(S.len.end(), 32 - lane, kCgPadding);
            S.off.push_back(S.off.back() + 32u * width);
        }
    }
    S.orig.insert(S.orig.end(), longs.begin(), longs.end());
    if (S.rows() >= (int64_t)kCgSelf) throw std::invalid_argument("problem too large for 27-bit CG positions");
    S.lrp.assign(1, 0);
    for (const uint32_t r : longs) S.lrp.push_back(S.lrp.back() + length(op, r));
}

// Contiguous runs of slices, one per virtual warp, of about equal work: a
// slice costs its stored entries (32 x its width) plus a fixed share; the long
// rows, which the warps take round-robin (row k: warp k mod nwarps), count
// toward their warp's share.  Warp w's run ends where the cumulative slice
// work comes nearest to (w + 1) x the average less the long-row work of warps
// 0..w (cumulative targets: the rounding of one warp does not carry into the
// next).
void split_slices(const PackedOperator &op, int64_t nwarps, CgSide &S) {
    const double fixed = 32.0 * 3.0;
    const int64_t ns = S.nslices();
    std::vector<double> extra(nwarps, 0.0);
    double total = 0.0;
    for (int64_t k = 0; k < S.nlong(); k++) {
        const double c = 32.0 * (double)((S.lrp[k + 1] - S.lrp[k] + 31) / 32) + fixed;
        extra[k % nwarps] += c;
        total += c;
    }
    std::vector<double> cum(ns + 1, 0.0);
    for (int64_t s = 0; s < ns; s++) cum[s + 1] = cum[s] + (double)(S.off[s + 1] - S.off[s]) + fixed;
    total += cum[ns];
    const double avg = total / (double)nwarps;
    S.split.assign(nwarps + 1, 0);
    double ce = 0.0;
    for (int64_t w = 0; w < nwarps; w++) {
        ce += extra[w];
        const double target = (double)(w + 1) * avg - ce;
        int64_t s = std::lower_bound(cum.begin(), cum.end(), target) - cum.begin();
        if (s > 0 && s <= ns && target - cum[s - 1] < cum[s] - target) s--;
        s = std::min<int64_t>(std::max<int64_t>(s, S.split[w]), ns);
        S.split[w + 1] = (uint32_t)s;
    }
    S.split[nwarps] = (uint32_t)ns;
}

// the rows' entries in stored order, each through map(entry word)
template <class M>
void fill(const PackedOperator &op, CgSide &S, M &&map) {
    const int64_t ns = S.nslices();
    S.ent.assign(S.off[ns], 0);
    S.lent.resize(S.lrp.back());
    for (int64_t r = 0; r < S.rows(); r++) {
        if (S.orig[r] == kNone) continue;
        uint32_t *e = r < 32 * ns ? S.ent.data() + S.off[r >> 5] + (r & 31) : S.lent.data() + S.lrp[r - 32 * ns];
        const uint32_t step = r < 32 * ns ? 32 : 1;
        for (uint32_t k = op.row_ptr[S.orig[r]]; k < op.row_ptr[S.orig[r] + 1]; k++, e += step)
            *e = (op.entries[k] & ~kColMask) | map(op.entries[k] & kColMask);
    }
}

std::vector<uint32_t> positions(const CgSide &S, int64_t n) {
    std::vector<uint32_t> pos(n, 0);
    for (int64_t r = 0; r < S.rows(); r++)
        if (S.orig[r] != kNone) pos[S.orig[r]] = (uint32_t)r;
    return pos;
}

// Dependent load rounds of each virtual warp's run as the kernel takes it
// (slices of at most `narrow` entries four at a time, wider ones alone, eight
// entries to a round); a virtual CTA counts the mean of its longest and its
// average warp.  Longest first, each to the least loaded CTA with room.
void place(CgSide &S, int nvirtual, int v, uint32_t narrow) {
    const int grid = (nvirtual + v - 1) / v;
    const int64_t nwarps = (int64_t)nvirtual * kCgVirtualWarps;
    std::vector<double> cost(nvirtual, 0.0);
    for (int c = 0; c < nvirtual; c++) {
        double sum = 0.0, most = 0.0;
        for (int w = 0; w < kCgVirtualWarps; w++) {
            const int64_t gw = (int64_t)c * kCgVirtualWarps + w;
            double r = 0.0;
            for (uint32_t s = S.split[gw]; s < S.split[gw + 1];) {
                uint32_t n = 0, width = 0;
                for (; n < 4 && s + n < S.split[gw + 1]; n++)
                    width = std::max(width, (S.off[s + n + 1] - S.off[s + n]) / 32);
                if (width <= narrow) {
                    r += 3.0;
                    s += n;
                } else {
                    r += 1.0 + 2.0 * (double)(((S.off[s + 1] - S.off[s]) / 32 + 7) / 8);
                    s++;
                }
            }
            for (int64_t l = gw; l < S.nlong(); l += nwarps) r += 1.0 + 2.0 * (double)((S.lrp[l + 1] - S.lrp[l] + 127) / 128);
            sum += r;
            most = std::max(most, r);
        }
        cost[c] = 0.5 * (most + sum / kCgVirtualWarps);
    }
    std::vector<int> order(nvirtual), count(grid, 0);
    for (int c = 0; c < nvirtual; c++) order[c] = c;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[a] > cost[b]; });
    std::vector<double> load(grid, 0.0);
    S.host.assign((size_t)grid * v, kNone);
    for (const int c : order) {
        int best = -1;
        for (int g = 0; g < grid; g++)
            if (count[g] < v && (best < 0 || load[g] < load[best])) best = g;
        S.host[(size_t)best * v + count[best]++] = (uint32_t)c;
        load[best] += cost[c];
    }
}

}  // namespace

CgTables build_cg_tables(const PackedOperator &A, const PackedOperator &AT, int nvirtual, int v) {
    const int64_t nwarps = (int64_t)nvirtual * kCgVirtualWarps;
    CgTables t;
    lay_out(A, t.dual);
    lay_out(AT, t.prim);
    split_slices(A, nwarps, t.dual);
    split_slices(AT, nwarps, t.prim);
    place(t.dual, nvirtual, v, 2);
    place(t.prim, nvirtual, v, 1);
    // singles: one entry in A^T, one in A, the same row and coefficient
    std::vector<uint8_t> seen(AT.nrows, 0), single(AT.nrows, 0);
    for (int64_t j = 0; j < A.nrows; j++)
        for (uint32_t k = A.row_ptr[j]; k < A.row_ptr[j + 1]; k++) {
            const uint32_t w = A.entries[k], i = w & kColMask;
            if (seen[i] < 2) seen[i]++;
            bool same = seen[i] == 1 && length(A, j) <= kCgLongRow && length(AT, i) == 1;
            if (same) {
                const uint32_t u = AT.entries[AT.row_ptr[i]];
                same = (int64_t)(u & kColMask) == j && !(u & kGroupFlag) &&
                       AT.palette[code_of(u)] == A.palette[code_of(w)];
            }
            single[i] = same;
        }
    const std::vector<uint32_t> dpos = positions(t.dual, A.nrows), ppos = positions(t.prim, AT.nrows);
    for (int64_t i = 0; i < AT.nrows; i++)
        if (single[i]) t.prim.len[ppos[i]] |= kCgSingle;
    fill(A, t.dual, [&](uint32_t i) { return single[i] ? kCgSelf : ppos[i]; });
    fill(AT, t.prim, [&](uint32_t j) { return dpos[j]; });
    // plain slices, marked last (the widths above come from unmarked offsets)
    for (int64_t s = 0; s < t.prim.nslices(); s++) {
        bool plain = true;
        for (int l = 0; l < 32; l++) plain = plain && t.prim.len[32 * s + l] == (1 | kCgSingle);
        if (plain) t.prim.off[s] |= kCgPlain;
    }
    for (int64_t s = 0; s < t.dual.nslices(); s++) {
        bool plain = true;
        for (int l = 0; l < 32; l++) {
            plain = plain && t.dual.len[32 * s + l] == 2;
            const uint32_t *e = t.dual.ent.data() + t.dual.off[s] + l;
            plain = plain && !((e[0] | e[32]) & kGroupFlag);
        }
        if (plain) t.dual.off[s] |= kCgPlain;
    }
    return t;
}

CgPlan plan_cg(const PackedOperator &A, const PackedOperator &AT, int sms) {
    CgPlan p;
    // Virtual CTAs of 512 threads: a row per thread, three to an SM at most.
    // They are spread over one CTA per SM; two of them run as one CTA,
    // without grid barriers.
    const int64_t want = (std::max(A.nrows, AT.nrows) + 511) / 512;
    p.nvirtual = (int)std::max<int64_t>(1, std::min<int64_t>(want, 3 * (int64_t)sms));
    p.v = p.nvirtual <= 2 ? p.nvirtual : (p.nvirtual + sms - 1) / sms;
    p.tables = build_cg_tables(A, AT, p.nvirtual, p.v);
    // Where the tables go: both passes' in shared memory if they fit, else in
    // turn in one region of it, else left in global memory.  us per CG iteration
    // with both / one region / streamed: 9 orbitals 12.0 / 11.9 / 16.8, 14: 16.0 /
    // 18.9 / 29.5, 16: 21.2 / 23.9 / 38.0, 8 with T2 23.7 / 26.5 / 31.1; 18, where
    // both just fit, 38.9 / 32.7 / 55.9 (the one size measured where one region
    // was the better).  Where both do not fit, one region / streamed: 19 orbitals
    // 65.1 / 71.8, 20: 48.3 / 64.8, 9 with T2 51.6 / 55.6.  Where neither fits,
    // streamed against the former kernel: 22 orbitals 95 (134), 24: 133 (195), 10
    // with T2 112 (177).
    auto words = [&](bool both) {   // of the CTA with most
        size_t most = 0;
        for (size_t c = 0; c < p.tables.dual.host.size() / p.v; c++) {
            size_t sum = 0;
            for (int w = 0; w < p.v * kCgVirtualWarps; w++) {
                size_t n[2] = {0, 0};
                int k = 0;
                for (const CgSide *s : {&p.tables.dual, &p.tables.prim}) {
                    const uint32_t vc = s->host[c * p.v + w / kCgVirtualWarps];
                    if (vc != kNone) {
                        const size_t gw = (size_t)vc * kCgVirtualWarps + w % kCgVirtualWarps;
                        n[k] = cg_table_words(s->split[gw + 1] - s->split[gw],
                                              s->at(s->split[gw + 1]) - s->at(s->split[gw]));
                    }
                    k++;
                }
                sum += both ? n[0] + n[1] : std::max(n[0], n[1]);
            }
            most = std::max(most, sum);
        }
        return most;
    };
    const size_t room = 227 * 1024 - kCgStaticSmem;
    p.in = kCgBoth;
    p.smem = 4 * words(true);
    if (p.smem > room && p.v == 3) {
        p.in = kCgOneRegion;
        p.smem = 4 * words(false);
    }
    if (p.smem > room) {
        p.in = kCgStreamed;
        p.smem = 0;
        if (p.v != 1) p.tables = build_cg_tables(A, AT, p.nvirtual, p.v = 1);
    }
    p.grid = (p.nvirtual + p.v - 1) / p.v;
    return p;
}

}  // namespace v2b
