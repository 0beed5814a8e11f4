// The on-chip schedule of a plan: its rows grouped into tasks, the tasks into dataflow levels,
// and its current planes packed into shared-memory slots by liveness.
//
// A task is what one lane runs for one point with its sums in registers: a source row, a
// destination's run of contribution rows (F_FIRST .. F_LAST) with the propagator that
// follows it on the same current, a propagator, an identity or clear over one current, or a
// destination amplitude's consecutive closures. Tasks of one level read nothing another task of
// that level writes, so the lanes of a point run them in any order; each current's and each
// amplitude's rows keep their order, so every value is the one the row order gives, bit for bit.
#pragma once
#include <stdint.h>

#include <string>
#include <vector>

#include "program.h"

namespace pacuda {

enum : uint32_t {
    F_WB = 8,        // the instruction's written values also go to the global arena
    F_ACC0 = 16,     // a closure whose parent 0 is the task's sums (its closing current, in registers)
    F_NOSTORE = 32,  // a destination run's last row keeps its sums in registers (no slot)
    F_TERM = 64,     // a closure that makes its amplitude from zero and stores its reduction term
};
struct Schedule {
    std::vector<Ins> ins;               // task instructions; operands are slots
    std::vector<uint32_t> task_first;   // tasks + 1 entries into ins
    std::vector<uint32_t> level_first;  // levels + 1 entries into tasks
    uint32_t cur_slots = 0;             // complex current slots per point
    uint32_t peak_live = 0;             // the most current slots live at one level (a floor for cur_slots)
    uint32_t amp_slots = 0;             // complex amplitude slots per point
    uint32_t terms = 0;                 // reduction terms per point (instead of amplitude slots)
    std::vector<uint32_t> loads;        // live-in currents: (global plane, slot, count) triples
    std::vector<uint32_t> amp_planes;   // per amplitude slot, its global amplitude plane
    std::vector<uint32_t> amp_slot_of;  // per global amplitude plane, its slot or ~0u
    uint32_t max_task_len = 0;
    std::vector<uint32_t> task_cost;    // per task, its algorithmic flops
    std::string why;                    // empty when the schedule exists
};

// The order in which a point's L lanes take a level's tasks: position j of a
// level goes to lane j % L, so each level is padded to whole rounds of L with ~0u (no task). The
// tasks of a level are assigned longest first to the least loaded lane.
void lane_order(const Schedule &s, uint32_t lanes, std::vector<uint32_t> &order, std::vector<uint32_t> &level_first);

// builds the schedule of a program; `forms` is the plan's momentum form count
bool build_schedule(const Program &p, uint32_t current_planes, uint32_t amplitude_planes, Schedule &out);

// For a run that only reduces its amplitudes (resolved from zero: offsets[outputs + 1], planes),
// when every amplitude gets exactly one closure row and feeds at most one of the reduction's
// terms: each closure row makes its amplitude from zero and stores its term (weight x |A|^2),
// and the points keep the terms (8 bytes each) instead of the amplitudes (16). False (the
// schedule unchanged) otherwise.
bool use_terms(Schedule &s, const uint32_t *offsets, const uint32_t *planes, uint32_t outputs, uint32_t amplitude_planes);

// The constants of a schedule's instructions, folded for the on-chip executor. A contribution
// multiplies its value by scale x factor, a propagator by a factor and the reciprocal of its form's
// norm, a closure's component by component factor x row factor: none of these depends on the point
// (the reciprocal depends on the form alone, and many currents share a form), so each product is
// an entry of a table that is computed once, and each reciprocal is computed once per form and
// point. A constant that is exactly real, exactly imaginary or one is marked as such: the executor
// then leaves out the products with its zero part.
enum FoldKind : uint32_t {
    FOLD_SCALE_FACTOR,   // scale[a] x factor[b]
    FOLD_FACTOR_FACTOR,  // factor[a] x factor[b]
    FOLD_FACTOR,         // factor[a]
    FOLD_MINUS_I,        // factor[a] x (0, -1)
};
enum FoldClass : uint32_t { C_REAL = 0, C_IMAG = 1, C_ONE = 2, C_GENERAL = 3 };
constexpr uint32_t kNoReciprocal = 0xffff;
// a position of a lane order without a task (beside it: an instruction that may be fetched)
constexpr uint32_t kNoTask = 0x80000000u;

// The executor's dispatch codes: the rows that plans are mostly made of, each with the class its
// constants have there, and everything else (by op and class).
enum RowCode : uint32_t {
    R_TENSOR_IMAG,  // op 4
    R_VECTOR_IMAG,  // op 6
    R_WEDGE_ONE,    // op 5
    R_CLOSE4_REAL,  // op 11 over 4 components of the task's sums, into a reduction term
    R_WEYL_A_REAL,  // op 2
    R_WEYL_B_REAL,  // op 3
    R_PROP_IMAG,    // op 9
    R_CLOSE2_REAL,  // op 11 over 2 components of the task's sums, into a reduction term
    R_OTHER = 15,
};
// pseudo op: the task's sums start from a destination's value (c its slot, s its components)
constexpr uint32_t kOpLoad = 0;

struct Folds {
    // The schedule's instructions with folded operands: a contribution's s is its entry; a
    // propagator's s is its reciprocal (kNoReciprocal: computed in place) and x its entry; an
    // identity's x is its entry; a closure's y is its components' first entry. An instruction's
    // class is in its head's count field. A destination run that adds to its destination's value is
    // preceded by a kOpLoad instruction (of kind K_CONTRIB).
    std::vector<Ins> ins;
    std::vector<uint32_t> task_first;   // tasks + 1 entries into ins
    std::vector<uint32_t> entries;      // (kind << 28 | a, b) per entry
    std::vector<uint32_t> reciprocals;  // per reciprocal, its form
};

// Folds a schedule. The scales and factors are read for the classes alone; without them (null: a
// program whose constants come with each call) every class is general.
void fold_constants(const Schedule &s, const double *scale_re, const double *scale_im, const double *factor_re,
                    const double *factor_im, Folds &out);
// the dispatch code of a folded instruction
uint32_t row_code(const Ins &i);

}  // namespace pacuda
