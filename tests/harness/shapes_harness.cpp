// Test harness (CPU): the product's launch shapes (pacuda_b200/csrc/shapes.h) driven from Python.
#include "../../pacuda_b200/csrc/shapes.h"

using namespace pacuda;

extern "C" {

// sizes: 5 numbers per plan (kept, bare, table, points, chosen); shapes: 2 per plan (points, keep).
// 1 when every plan fits, with the bytes kept for folded entries in *table, else 0
int shapes(const uint64_t *sizes, uint32_t plans, int threads, uint64_t room, int spread, uint64_t *table, uint32_t *out) {
    std::vector<PlanSize> p(plans);
    for (uint32_t k = 0; k < plans; k++) {
        p[k].kept = sizes[5 * k];
        p[k].bare = sizes[5 * k + 1];
        p[k].table = sizes[5 * k + 2];
        p[k].points = (uint32_t)sizes[5 * k + 3];
        p[k].chosen = sizes[5 * k + 4] != 0;
    }
    size_t kept = 0;
    std::vector<PlanShape> s;
    if (!launch_shapes(p, threads, room, spread != 0, kept, s)) return 0;
    *table = kept;
    for (uint32_t k = 0; k < plans; k++) {
        out[2 * k] = s[k].points;
        out[2 * k + 1] = s[k].keep;
    }
    return 1;
}
}
