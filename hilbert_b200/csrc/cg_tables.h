// The constraint operator as the conjugate-gradient kernel reads it.
#pragma once

#include <cstdint>
#include <vector>

#include "v2rdm_problem.h"

#ifdef __CUDACC__
#define V2B_HD __host__ __device__
#else
#define V2B_HD
#endif

namespace v2b {

// The rows of A (dual side) and of A^T (primal side) in SELL-C-sigma form,
// C = 32: rows of at most kCgLongRow entries, sorted by length inside windows
// of kCgSigma rows (longest first, stable), in slices of 32 rows stored
// column-major (entry k of the slice's lane l at off[s] + 32 k + l).  The
// kernel keeps its vectors in this order: position 32 s + l for lane l of
// slice s, position 32 nslices + l for long row l, and the entries' columns
// are positions of the other side, so a row's own values are read and written
// without an index.
//   entry: bits 0..26 position, 27..30 palette index, 31 group flag
//   len:   bits 0..5 entries of the row (kCgPadding on padding), bit 7 kCgSingle
// A primal variable with one entry in A^T and one in A, of the same coefficient
// (a Q2, G2, T2, ... element in its own defining row: 84% of the (20e,20o) DQG
// variables), is a "single": its constraint forms t = coef * p from its own p, the entry
// (position kCgSelf) needs no gather, and t is not stored.
//
// split[w] .. split[w + 1] - 1 are the slices of virtual warp w, long rows
// w, w + nwarps, ... its long rows.  The virtual warps (16 to a virtual CTA)
// define the order of the CG's dot products; which thread does the work does
// not show in the result.
constexpr uint32_t kCgLongRow = 32;
constexpr int64_t kCgSigma = 8192;
constexpr uint32_t kCgSelf = (1u << 27) - 1u;
constexpr uint8_t kCgSingle = 0x80, kCgPadding = 0x7f;
// a slice without padding whose rows are all singles (primal side), or all
// have two entries and no group flag (dual side): 84% and 75% of (20e,20o)
constexpr uint32_t kCgPlain = 1u;
constexpr int kCgVirtualWarps = 16;   // virtual warps of a virtual CTA (512 threads)

struct CgSide {
    // slices: offsets (nslices + 1; multiples of 32, bit 0 kCgPlain), entries
    std::vector<uint32_t> off, ent;
    std::vector<uint8_t> len;            // 32 nslices
    std::vector<uint32_t> lrp, lent;     // long rows: offsets (nlong + 1), entries
    std::vector<uint32_t> split;         // nwarps + 1
    std::vector<uint32_t> orig;          // original row per position, 0xffffffff on padding
    std::vector<uint32_t> host;          // V per CTA: the virtual CTAs it hosts, 0xffffffff for none
    uint32_t at(int64_t s) const { return off[s] & ~kCgPlain; }
    int64_t nslices() const { return (int64_t)off.size() - 1; }
    int64_t nlong() const { return (int64_t)lrp.size() - 1; }
    int64_t rows() const { return (int64_t)orig.size(); }
};
struct CgTables {
    CgSide dual, prim;
};

// A virtual warp's run of slices b .. e - 1 and where the CG kernel finds its
// tables in shared memory: entries, then lengths, then slice offsets.
struct CgRun {
    uint32_t b, e, gw;   // slices; the virtual warp, 0xffffffff for none
    uint32_t off;        // word of slice b's offset
    // word where entry 0 of the side would stand: below 0 for most runs, and
    // signed, so that base + ent + index is the entry's word as a 64-bit address
    int32_t ent;
    uint32_t len;        // byte of slice b's lengths
};
// the words of a run's tables
V2B_HD inline uint32_t cg_table_words(uint32_t nslices, uint32_t nent) {
    return nent + 8u * nslices + ((nslices + 4u) & ~3u);
}
// the run's tables from word `at` on; its entries are e0 .. e0 + ne - 1
V2B_HD inline void cg_place_run(CgRun &r, uint32_t at, uint32_t e0, uint32_t ne) {
    r.ent = (int32_t)(at - e0);
    r.len = 4u * (at + ne);
    r.off = at + ne + 8u * (r.e - r.b);
}

// nvirtual virtual CTAs, v of them to a CTA (grid = ceil(nvirtual / v)).  Which
// CTA hosts a virtual CTA is free, and chosen per side so that the CTAs' work
// between two barriers is even: a run of wide rows takes longer than its
// entries say (its loads come in dependent rounds), and neighbours are alike.
CgTables build_cg_tables(const PackedOperator &A, const PackedOperator &AT, int nvirtual, int v);

// Where the CG kernel reads its tables: shared memory, both passes' side by
// side or in turn in one region, or global memory.
enum CgTablesIn { kCgBoth, kCgOneRegion, kCgStreamed };
constexpr size_t kCgStaticSmem = 4096;   // at least the kernel's static shared memory
struct CgPlan {
    CgTables tables;
    int nvirtual, v, grid;
    CgTablesIn in;
    size_t smem;   // dynamic shared memory of a CTA
};
CgPlan plan_cg(const PackedOperator &A, const PackedOperator &AT, int sms);

}  // namespace v2b
