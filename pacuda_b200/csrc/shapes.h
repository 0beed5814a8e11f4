// How a launch of the on-chip executor keeps its plans in shared memory (host code without CUDA).
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

namespace pacuda {

// points per block: 1 .. kMaxPoints; a point then has warps * floor(32 / P) lanes (a lane of all
// P points is P adjacent threads of one warp)
constexpr uint32_t kMaxPoints = 32;

// whether a block of `threads` runs `points` points within `max_smem` bytes
inline bool tiled_points_fit(uint32_t points, size_t point_bytes, int threads, size_t max_smem) {
    return points >= 1 && points <= kMaxPoints && threads >= 32 && (size_t)points * point_bytes <= max_smem;
}

// the most points per block that fit, or 0
inline uint32_t tiled_max_points(size_t point_bytes, int threads, size_t max_smem) {
    for (uint32_t np = kMaxPoints; np >= 1; np--)
        if (tiled_points_fit(np, point_bytes, threads, max_smem)) return np;
    return 0;
}

// the default points per block: of those that fit, the count that leaves the fewest threads of a
// warp without a lane (P * floor(32 / P) largest), the larger on ties; 0 when none fits
inline uint32_t tiled_default_points(size_t point_bytes, int threads, size_t max_smem) {
    uint32_t best = 0;
    for (uint32_t np = 1; np <= kMaxPoints; np++)
        if (tiled_points_fit(np, point_bytes, threads, max_smem) && (!best || np * (32 / np) >= best * (32 / best)))
            best = np;
    return best;
}

// What a plan asks of a launch: the bytes of one point with its forms' reciprocals and without
// (`bare`), of its table of folded entries, and the points per block that it has (0: the default),
// `chosen` when the caller or the tuner chose them.
struct PlanSize {
    size_t kept = 0, bare = 0, table = 0;
    uint32_t points = 0;
    bool chosen = false;
};
struct PlanShape {
    uint32_t points = 0;
    bool keep = true;  // whether its points keep their reciprocals
};

// The shapes of a launch's plans in blocks of `threads` with `room` bytes of shared memory, and the
// bytes that a block keeps for folded entries (`table`: the largest plan's, or none: the entries are then
// read from global memory). Entries and reciprocals save work where there is room for them (a point's
// reciprocals are 80 of 11 440 bytes in qg>qgg, a table 144); neither may cost a launch that fits without
// them: one point of every plan, and the points per block that were chosen for it. `spread`: one point
// per block whatever was chosen. False when a plan's point does not fit.
inline bool launch_shapes(const std::vector<PlanSize> &plans, int threads, size_t room, bool spread, size_t &table,
                          std::vector<PlanShape> &out) {
    table = 0;
    for (const PlanSize &p : plans) table = std::max(table, p.table);
    for (const PlanSize &p : plans) {
        auto fits = [&](uint32_t n) { return table <= room && tiled_points_fit(n, p.bare, threads, room - table); };
        const bool chosen = p.chosen && !spread && tiled_points_fit(p.points, p.bare, threads, room);
        if (!fits(chosen ? p.points : 1)) table = 0;
    }
    out.assign(plans.size(), PlanShape());
    for (size_t k = 0; k < plans.size(); k++) {
        const PlanSize &p = plans[k];
        const size_t left = room - table;
        PlanShape &s = out[k];
        if (spread) s.points = 1;
        else if (tiled_points_fit(p.points, p.chosen ? p.bare : p.kept, threads, left)) s.points = p.points;
        else s.points = tiled_default_points(p.kept, threads, left);
        if (!s.points) s.points = tiled_default_points(p.bare, threads, left);
        s.keep = tiled_points_fit(s.points, p.kept, threads, left);
        if (!tiled_points_fit(s.points, p.bare, threads, left)) return false;
    }
    return true;
}

}  // namespace pacuda
