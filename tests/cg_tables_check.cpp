// Prints, for the CG tables of one problem, how far each run's words lie from
// where the kernel looks for them (0 0: every entry, offset and length is
// found inside its run's own words), then the form that the kernel takes on 148 SMs.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "cg_tables.h"

using namespace v2b;

// the kernel forms base + r.ent as a 64-bit address and adds the entry's index
static int64_t entry_word(const CgRun &r, uint32_t k) { return (int64_t)r.ent + (int64_t)k; }

int main(int argc, char **argv) {
    ProblemSpec spec;
    spec.nmo = atoi(argv[1]);
    spec.nalpha = atoi(argv[2]);
    spec.nbeta = atoi(argv[3]);
    spec.positivity = atoi(argv[4]) & 15;
    spec.constrain_d3 = atoi(argv[4]) & 16;
    spec.doci = argc > 5 && !strcmp(argv[5], "doci");
    const Problem p = make_problem(spec);
    const PackedOperator A = build_A(p), AT = build_AT(p);
    const CgPlan plan = plan_cg(A, AT, 148);
    const CgTables &t = plan.tables;
    const int v = plan.v, grid = plan.grid;
    long runs = 0, wrong = 0;
    for (const bool shared : {false, true})
        for (int c = 0; c < grid; c++) {
            uint32_t at = 0;
            for (int w = 0; w < v * kCgVirtualWarps; w++) {
                uint32_t most = 0;
                for (const CgSide *s : {&t.dual, &t.prim}) {
                    const uint32_t vc = s->host[(size_t)c * v + w / kCgVirtualWarps];
                    if (vc == 0xffffffffu) continue;
                    CgRun r{};
                    r.gw = vc * kCgVirtualWarps + w % kCgVirtualWarps;
                    r.b = s->split[r.gw];
                    r.e = s->split[r.gw + 1];
                    const uint32_t e0 = s->at(r.b), ne = s->at(r.e) - e0, n = r.e - r.b;
                    const uint32_t words = cg_table_words(n, ne), from = shared ? at : at + most;
                    cg_place_run(r, from, e0, ne);
                    runs++;
                    bool ok = r.len % 16 == 0 && (from + 0u) % 4 == 0;
                    for (uint32_t i = r.b; i < r.e; i++)
                        for (uint32_t k = s->at(i); k < s->at(i + 1); k++)
                            ok = ok && entry_word(r, k) >= from && entry_word(r, k) < (int64_t)from + ne;
                    ok = ok && r.len >= 4 * (from + ne) && r.len + 32 * n <= 4 * r.off;
                    ok = ok && r.off + n + 1 <= from + words;
                    wrong += !ok;
                    most = shared ? std::max(most, words) : most + words;
                }
                at += most;
            }
        }
    printf("%ld runs, %ld wrong\n", runs, wrong);
    const char *names[] = {"both", "one region", "streamed"};
    printf("%d per CTA, %s, %zu bytes\n", v, names[plan.in], plan.smem);
    return 0;
}
