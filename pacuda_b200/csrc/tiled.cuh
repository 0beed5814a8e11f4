// The on-chip executor: a persistent kernel whose blocks take groups of points; each point's
// currents, amplitudes and forms live in shared-memory slots (schedule.h), a point's lanes run
// the tasks of one dataflow level at a time, and nothing but the external momenta comes in and
// the outputs go out (in the C ABI's mode also the arena's live-in planes in and its written
// planes out).
//
// A block runs P points at once (1 .. 32). A lane of all P points is a group of P adjacent
// threads of one warp (floor(32 / P) groups per warp, the warp's other threads idle), so each
// point has G = warps * floor(32 / P) lanes. The P threads of a group run the same task on
// consecutive points: their instruction fetches are one broadcast, their shared-memory values
// ([slot][P], interleaved) are contiguous, and their global stores cover P consecutive points of
// a plane. All points take the same lane order, so a block's points move through the levels
// together and meet at the block's barrier. A block takes one work item at a time: one plan's
// next P points. An SM runs 1 to 16 such blocks (each with its share of the warps and shared
// memory), which reach their barriers at different times; batch blocks of 1 and 8 points run a
// copy of the levels with that count built in (run_levels over SlotView<K, ABI, NP>).
#pragma once
#include <stdint.h>

#include "arith.cuh"
#include "executor.cuh"
#include "program.h"
#include "schedule.h"

namespace pacuda {

struct TiledPlan {
    // the schedule (instructions in the 16-byte form: pack_ins)
    const uint4 *ins;
    const uint32_t *order;        // per level position, its task's first instruction; lane = position % G
    const uint32_t *level_first;  // levels + 1 entries into order
    uint32_t levels;
    uint32_t cur_slots, amp_slots, forms;
    uint32_t terms;               // reduction terms kept instead of amplitudes (batch mode), or 0
    uint32_t points;              // P points per block
    uint32_t lanes;               // G lanes per point: warps * floor(32 / P)
    uint32_t point_bytes;         // shared memory of one point
    // constants: f64 (sources); the folded entries in the kind's values (rows: schedule.h Folds)
    const double *s64, *f64;
    const void *folded;
    uint32_t entries;             // folded entries, and how many of them a block keeps in shared memory
    uint32_t near;                // (all, or where they do not fit none)
    uint32_t factors;
    // the C ABI's mode: the constants come with the call, and a block folds its near entries itself
    const uint32_t *entry_list;
    const void *kconst;
    uint32_t scales;
    // the forms whose reciprocal norms a point keeps
    const uint32_t *recip_forms;
    uint32_t recips;
    // forms from external momenta (source-major planes of `points` values per point)
    const uint32_t *form_terms, *term_slots;
    const double *coefficients;
    // the resolved reduction (batch mode): outputs, offsets into (slot, weight) pairs
    const uint32_t *red_offsets, *red_slots;
    const double *red_weights;
    uint32_t outputs;
    // the C ABI's mode: live-in current planes, the amplitude slots' planes
    const uint32_t *loads;
    uint32_t nloads;
    const uint32_t *amp_planes;
};

// one launch: plans (a batch) and, per plan, its points
struct TiledLaunch {
    const TiledPlan *plans;
    uint32_t nplans;
    const unsigned long long *item_first;  // nplans + 1 prefix sums of work items (a block's points)
    const double *const *external;         // per plan: source-major planes [(leg * 4 + k) * count + i]
    const uint32_t *count;                 // per plan: its points
    double *const *output;                 // per plan: [point][outputs] (batch mode)
    unsigned long long *counter;           // work-item counter (zeroed before the launch)
    // the C ABI's mode (one plan): the arenas in the kind's layout, stride ld
    bool abi;
    void *cre, *cim, *are, *aim;
    const double *mom;                     // uploaded forms (f64 planes), or null
    size_t ld;
    uint32_t const_bytes;                  // shared memory kept for a plan's folded entries
    bool far;                              // a plan has more entries than 16 bits index
};

// The on-chip executor's 16-byte instruction: a head, the forms' bytes, then (a, b), (c, s), (x, y)
// as 16-bit pairs. Every field of a plan whose points fit shared memory fits (slots and constant
// indices below 65536, forms below 256); the host checks. An entry's index, which a plan with many pairs
// of constants may need more bits for, has its upper half in a field that its row does not use. The
// head's sixteen bits:
constexpr uint32_t H_CODE = 15;        // RowCode
constexpr uint32_t H_CLASS = 3 << 4;   // FoldClass
constexpr uint32_t H_END = 1 << 6;     // the task's last instruction
constexpr uint32_t H_STORE = 1 << 7;   // a contribution that stores its sums to their slots
constexpr uint32_t H_OP = 15 << 8;
constexpr uint32_t H_ACC0 = 1 << 12, H_TERM = 1 << 13;  // F_ACC0, F_TERM
constexpr uint32_t H_SET = 1 << 14;    // a contribution that sets its sums (the C ABI's mode)
constexpr uint32_t H_WB = 1 << 15;     // F_WB of an instruction that writes
// or-ed into every head, it makes each row one of R_OTHER with general constants
constexpr uint32_t H_PLAIN = H_CODE | H_CLASS;

struct Row16 {
    uint4 w;
    __device__ __forceinline__ uint32_t op() const { return w.x >> 8 & 15; }
    __device__ __forceinline__ uint32_t cls() const { return w.x >> 4 & 3; }
    __device__ __forceinline__ uint32_t f0() const { return w.x >> 16 & 0xff; }
    __device__ __forceinline__ uint32_t f1() const { return w.x >> 24; }
    __device__ __forceinline__ uint32_t a() const { return w.y & 0xffff; }
    __device__ __forceinline__ uint32_t b() const { return w.y >> 16; }
    __device__ __forceinline__ uint32_t c() const { return w.z & 0xffff; }
    __device__ __forceinline__ uint32_t s() const { return w.z >> 16; }
    __device__ __forceinline__ uint32_t x() const { return w.w & 0xffff; }
    __device__ __forceinline__ uint32_t y() const { return w.w >> 16; }
    // the entry of a contribution (s, x), a propagator or identity (x, c), a closure's first (y, x)
    __device__ __forceinline__ uint32_t entry_s() const { return __byte_perm(w.z, w.w, 0x5432); }
    __device__ __forceinline__ uint32_t entry_x() const { return __byte_perm(w.w, w.z, 0x5410); }
    __device__ __forceinline__ uint32_t entry_y() const { return __byte_perm(w.w, 0, 0x1032); }
};

// a hint: the line holding `p` into L1 (no register waits for it)
__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// a complex value as shared memory holds it: (re, im) side by side, one 8- or 16-byte access
template <class R> struct alignas(2 * sizeof(R)) Pair {
    R re, im;
};

// a pair through the read-only path
template <class R> __device__ __forceinline__ Pair<R> ldg_pair(const Pair<R> *p) {
    union {
        uint4 w4;
        uint2 w2;
        Pair<R> v;
    } u;
    if (sizeof(Pair<R>) == 16) u.w4 = __ldg(reinterpret_cast<const uint4 *>(p));
    else u.w2 = __ldg(reinterpret_cast<const uint2 *>(p));
    return u.v;
}

__device__ __forceinline__ double to_f64_value(double x) { return x; }
__device__ __forceinline__ double to_f64_value(D x) { return __dadd_rn((double)x.hi, (double)x.lo); }

// the C ABI's mode: where an item's points write their planes back (thread 0 sets it per item;
// in shared memory so that no lane holds these in registers through its tasks)
struct AbiItem {
    void *cre, *cim;
    size_t ld;
    unsigned long long first;  // the item's first point
    uint32_t count;            // the plan's points
};
static __shared__ AbiItem abi_item;

// NP: the block's points when known at compile time (0: np at run time); with NP a slot's
// address is a shift of its index and its components' addresses constant offsets from it.
// FAR: a table of more entries than 16 bits index
template <class K, bool ABI, int NP = 0, bool FAR = false> struct SlotView {
    typedef typename K::R R;
    typedef typename K::Den Den;
    typedef typename K::Amp Amp;
    typedef typename K::Const Const;
    Pair<R> *cur_;        // [slot][points of the region]
    Pair<Amp> *amp_;      // [amplitude slot][points of the region]
    double *term_;        // [reduction term][points] (a schedule that keeps terms)
    const Den *mom;
    const R *rec_;        // [reciprocal][points]
    const Pair<R> *folded_;  // the plan's folded entries (in shared memory where NP is known)
    uint32_t np, pw;      // the block's points (interleaved) and this thread's
    static constexpr int kPoints = NP;
    // a row's entry
    __device__ __forceinline__ uint32_t entry_s(const Row16 &o) const { return FAR ? o.entry_s() : o.s(); }
    __device__ __forceinline__ uint32_t entry_x(const Row16 &o) const { return FAR ? o.entry_x() : o.x(); }
    __device__ __forceinline__ uint32_t entry_y(const Row16 &o) const { return FAR ? o.entry_y() : o.y(); }
    __device__ __forceinline__ uint32_t at(uint32_t slot) const { return NP ? slot * NP + pw : slot * np + pw; }
    // the same view with the addressing of N points per block (valid when np == N)
    // and its entries at `near` in shared memory
    template <int N> __device__ __forceinline__ SlotView<K, ABI, N> with_points(const Pair<R> *near) const {
        SlotView<K, ABI, N> o;
        o.cur_ = cur_;
        o.amp_ = amp_;
        o.term_ = term_;
        o.mom = mom;
        o.rec_ = rec_;
        o.folded_ = near;
        o.np = N;
        o.pw = pw;
        return o;
    }
    __device__ __forceinline__ Cx<R> cur(uint32_t slot) const {
        Pair<R> v = cur_[at(slot)];
        return cx(v.re, v.im);
    }
    __device__ __forceinline__ void put(uint32_t slot, Cx<R> v) const {
        Pair<R> x;
        x.re = v.re;
        x.im = v.im;
        cur_[at(slot)] = x;
    }
    // the four components of a form (side by side in blocks of one point: two 16-byte loads)
    __device__ __forceinline__ void form(uint32_t f, Den (&q)[4]) const {
        if (NP == 1) {
            const Pair<Den> *p = reinterpret_cast<const Pair<Den> *>(mom + f * 4);
            const Pair<Den> x = p[0], y = p[1];
            q[0] = x.re;
            q[1] = x.im;
            q[2] = y.re;
            q[3] = y.im;
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++) q[k] = mom[at(f * 4 + k)];
        }
    }
    __device__ __forceinline__ R reciprocal(uint32_t r) const { return rec_[at(r)]; }
    __device__ __forceinline__ Cx<R> folded(uint32_t n) const {
        const Pair<R> v = folded_[n];
        return cx(v.re, v.im);
    }
    __device__ __forceinline__ void amp(uint32_t a, Amp &re, Amp &im) const {
        Pair<Amp> v = amp_[at(a)];
        re = v.re;
        im = v.im;
    }
    // a reduction term: fma(re, re, im x im), which the reduction multiplies by its weight
    __device__ __forceinline__ void put_term(uint32_t t, Amp re, Amp im) const {
        double r = to_f64_value(re), i = to_f64_value(im);
        term_[at(t)] = __fma_rn(r, r, __dmul_rn(i, i));
    }
    __device__ __forceinline__ void put_amp(uint32_t a, Amp re, Amp im) const {
        Pair<Amp> x;
        x.re = re;
        x.im = im;
        amp_[at(a)] = x;
    }
    __device__ __forceinline__ void writeback(uint32_t plane, const Cx<R> *v, int n) const {
        if (ABI) {
            const unsigned long long point = abi_item.first + pw;
            if (point < abi_item.count) {
                R *re = (R *)abi_item.cre, *im = (R *)abi_item.cim;
                const size_t ld = abi_item.ld;
                for (int k = 0; k < n; k++) {
                    re[(plane + k) * ld + point] = v[k].re;
                    im[(plane + k) * ld + point] = v[k].im;
                }
            }
        }
    }
};

// ---- rows on folded constants ----------------------------------------------------------------
// What a row costs is FP64 (or f32) instructions, and a third of what the plain formulas spend goes
// to constants: a scale that is i g has a zero real part, a closure's component factors are +-1, a
// propagator of -i times a real factor is imaginary. The rows below take the folded constants
// (schedule.h) with their classes: products with an exactly zero part are left out. The values
// are the plain formulas' in every bit for finite operands, except that a zero may have the other
// sign; no later operation of a plan makes anything but a zero's sign of that, and a reduced output
// has none. Where an operand is not finite the plain formulas' 0 x inf makes a NaN; such a
// point's outputs are not finite on this path either (every component that enters a row still
// enters it), and the point is computed again with the plain formulas (`plain`). The C ABI's mode, whose currents and amplitudes leave the block, always uses those.
// What bounds the executor is the instructions of a row (fetch, decode, moves, tests beside the
// arithmetic) and their latency with 16 warps per SM, so the common rows each have a dispatch code
// and straight code without class or flag tests: of gg>ggg's 22 900 warp instructions per point,
// 12 600 of them FP64, 17 200 and 10 150 are left. Measured on B200, 4096 points of gg>ggg: 173 ->
// 146 us; 50 021 of qg>qgg with contracted multiply-adds: 430 -> 374 us; 65 537 of the 3-jet mix in
// df64, where every product left out is about ten f32 instructions: 10.6 -> 6.95 ms. (The folded
// constants alone, with class and flag tests in every row: no gain in f64.)

// acc += val times an entry of class CLS: each class adds to the sums in place (a value that met the
// others' at a join would cost two register moves per f64)
template <int CLS, int N, class R>
__device__ __forceinline__ void add_folded(Cx<R> *acc, const Cx<R> (&val)[N], Cx<R> s) {
#pragma unroll
    for (int k = 0; k < N; k++) {
        if (CLS == (int)C_IMAG) acc[k] = cx(acc[k].re - val[k].im * s.im, acc[k].im + val[k].re * s.im);
        else if (CLS == (int)C_ONE) acc[k] = acc[k] + val[k];
        else if (CLS == (int)C_REAL) acc[k] = cx(acc[k].re + val[k].re * s.re, acc[k].im + val[k].im * s.re);
        else acc[k] = acc[k] + val[k] * s;
    }
}

constexpr int kClassOfRow = -1;  // the class is in the row

// A destination's sums start at zero (a batch's task), so a run's first row adds like the others;
// the C ABI's mode, where a zero's sign is seen, starts them with the first row's value.
template <class K, int OP, int CLS, bool ABI, class V>
__device__ __forceinline__ void tile_contribution(const V &v, const Row16 &o, Cx<typename K::R> *acc) {
    typedef typename K::R R;
    typedef typename K::Den Den;
    constexpr int c0 = Shape<OP>::c0, c1 = Shape<OP>::c1, cd = Shape<OP>::cd;
    Cx<R> l[c0], r[c1], val[cd], scale = cx(konst<R>(1.0), konst<R>(0.0));
    R q0[4], q1[4];
    const uint32_t a = o.a(), b = o.b();
    if (CLS != (int)C_ONE) scale = v.folded(v.entry_s(o));
#pragma unroll
    for (int k = 0; k < c0; k++) l[k] = v.cur(a + k);
#pragma unroll
    for (int k = 0; k < c1; k++) r[k] = v.cur(b + k);
    if (OP == 6) {
        Den d0[4], d1[4];
        v.form(o.f0(), d0);
        v.form(o.f1(), d1);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            q0[k] = form_as<R>(d0[k]);
            q1[k] = form_as<R>(d1[k]);
        }
    }
    contribution<OP>(l, r, q0, q1, val);
    if (ABI && (o.w.x & H_SET)) {
#pragma unroll
        for (int k = 0; k < cd; k++) acc[k] = val[k] * scale;
    } else if (CLS != kClassOfRow) {
        add_folded<CLS>(acc, val, scale);
    } else {
        const uint32_t cls = ABI ? (uint32_t)C_GENERAL : o.cls();
        if (cls == C_IMAG) add_folded<C_IMAG>(acc, val, scale);
        else if (cls == C_GENERAL) add_folded<C_GENERAL>(acc, val, scale);
        else add_folded<C_REAL>(acc, val, scale);  // (one among them)
    }
    if (o.w.x & H_STORE) {
        const uint32_t c = o.c();
#pragma unroll
        for (int k = 0; k < cd; k++) v.put(c + k, acc[k]);
    }
    if (ABI && (o.w.x & H_WB)) v.writeback(o.y(), acc, cd);
}

// 1 / (q . q) of a form in the kind's values
template <class K> __device__ __forceinline__ typename K::R form_reciprocal(const typename K::Den (&q)[4]) {
    typedef typename K::Den Den;
    Den norm = ((q[0] * q[0] - q[1] * q[1]) - q[2] * q[2]) - q[3] * q[3];
    return den_real(konst<Den>(1.0) / norm, (typename K::R *)nullptr);
}

template <class K, int OP, bool ABI, class V>
__device__ __forceinline__ void tile_propagator(const V &v, const Row16 &o) {
    typedef typename K::R R;
    typedef typename K::Den Den;
    constexpr int m = OP == 9 ? 4 : 2;
    const uint32_t a = o.a();
    Den q[4];
    R reciprocal;
    if (o.s() != kNoReciprocal) {
        reciprocal = v.reciprocal(o.s());
        if (OP != 9) v.form(o.f0(), q);
    } else {
        v.form(o.f0(), q);
        reciprocal = form_reciprocal<K>(q);
    }
    const Cx<R> s = scaled(v.folded(v.entry_x(o)), reciprocal);
    Cx<R> c[m], out[m];
#pragma unroll
    for (int k = 0; k < m; k++) out[k] = v.cur(a + k);
    if (OP != 9) {
        R p[4];
#pragma unroll
        for (int k = 0; k < 4; k++) p[k] = form_as<R>(q[k]);
#pragma unroll
        for (int k = 0; k < m; k++) c[k] = out[k];
        weyl_slash<OP>(c, p, out);
    }
    const uint32_t cls = ABI ? (uint32_t)C_GENERAL : o.cls();
    if (cls == C_IMAG) {
#pragma unroll
        for (int k = 0; k < m; k++) v.put(a + k, cx(-(out[k].im * s.im), out[k].re * s.im));
    } else if (cls != C_GENERAL) {  // (a unit factor's s is the reciprocal)
#pragma unroll
        for (int k = 0; k < m; k++) v.put(a + k, scaled(out[k], s.re));
    } else {
#pragma unroll
        for (int k = 0; k < m; k++) {
            out[k] = out[k] * s;
            v.put(a + k, out[k]);
        }
        if (ABI && (o.w.x & H_WB)) v.writeback(o.y(), out, m);
    }
}

// op 9 with an imaginary constant and a kept reciprocal
template <class K, class V> __device__ __forceinline__ void tile_vector_propagator(const V &v, const Row16 &o) {
    typedef typename K::R R;
    const uint32_t a = o.a();
    const R s = v.folded(v.entry_x(o)).im * v.reciprocal(o.s());
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const Cx<R> c = v.cur(a + k);
        v.put(a + k, cx(-(c.im * s), c.re * s));
    }
}

// a closure's component added to its amplitude: (l r) times its entry
template <bool REAL, class R, class A>
__device__ __forceinline__ void add_closure(Cx<R> l, Cx<R> r, Cx<R> s, A &dr, A &di) {
    const R pr = l.re * r.re - l.im * r.im, pi = l.re * r.im + l.im * r.re;
    if (REAL) {
        dr = dr + amp_of(pr * s.re, (A *)nullptr);
        di = di + amp_of(pi * s.re, (A *)nullptr);
    } else {
        dr = dr + amp_of(pr * s.re - pi * s.im, (A *)nullptr);
        di = di + amp_of(pr * s.im + pi * s.re, (A *)nullptr);
    }
}

// a closure of N components of the task's sums with real constants, into its reduction term
template <class K, int N, class V>
__device__ __forceinline__ void tile_closure_term(const V &v, const Row16 &o, const Cx<typename K::R> *acc) {
    typedef typename K::Amp Amp;
    Amp dr = konst<Amp>(0.0), di = konst<Amp>(0.0);
    const uint32_t b = o.b(), y = v.entry_y(o);
#pragma unroll
    for (int k = 0; k < N; k++) add_closure<true>(acc[k], v.cur(b + k), v.folded(y + k), dr, di);
    v.put_term(o.c(), dr, di);
}

template <class K, class V>
__device__ __forceinline__ void tile_closure(const V &v, const Row16 &o, const Cx<typename K::R> *acc) {
    typedef typename K::Amp Amp;
    Amp dr, di;
    const bool term = o.w.x & H_TERM;
    if (term) {  // the amplitude's only closure, from zero
        dr = konst<Amp>(0.0);
        di = konst<Amp>(0.0);
    } else {
        v.amp(o.c(), dr, di);
    }
    const uint32_t a = o.a(), b = o.b(), n = o.s(), y = v.entry_y(o);
    if (o.w.x & H_ACC0) {
        // parent 0 is the task's sums (at most 6 components): indices known at compile time keep
        // the sums in registers
#pragma unroll
        for (int k = 0; k < 6; k++) {
            if ((uint32_t)k >= n) break;
            add_closure<false>(acc[k], v.cur(b + k), v.folded(y + k), dr, di);
        }
    } else {
        for (uint32_t k = 0; k < n; k++) add_closure<false>(v.cur(a + k), v.cur(b + k), v.folded(y + k), dr, di);
    }
    if (!term) v.put_amp(o.c(), dr, di);
    else if (o.c() != 0xffff) v.put_term(o.c(), dr, di);
}

// identity (op 10) and clear (op 1) over `b` components
template <class K, class V> __device__ __forceinline__ void tile_identity(const V &v, const Row16 &o) {
    typedef typename K::R R;
    const Cx<R> f = v.folded(v.entry_x(o));
    for (uint32_t k = 0; k < o.b(); k++) {
        Cx<R> x = times_factor(f.re, f.im, v.cur(o.a() + k));
        v.put(o.a() + k, x);
        if (o.w.x & H_WB) v.writeback(o.y() + k, &x, 1);
    }
}
template <class K, class V> __device__ __forceinline__ void tile_clear(const V &v, const Row16 &o) {
    typedef typename K::R R;
    Cx<R> z = cx(konst<R>(0.0), konst<R>(0.0));
    for (uint32_t k = 0; k < o.b(); k++) {
        v.put(o.a() + k, z);
        if (o.w.x & H_WB) v.writeback(o.y() + k, &z, 1);
    }
}

// the task's sums from a destination's value
template <class K, class V> __device__ __forceinline__ void tile_load(const V &v, const Row16 &o, Cx<typename K::R> *acc) {
    const uint32_t c = o.c(), n = o.s();
    acc[0] = v.cur(c);
    acc[1] = v.cur(c + 1);
    if (n > 2) {
        acc[2] = v.cur(c + 2);
        acc[3] = v.cur(c + 3);
    }
    if (n > 4) {
        acc[4] = v.cur(c + 4);
        acc[5] = v.cur(c + 5);
    }
}

// one row of any op but a source, its sum kept in `acc` across a destination's run: the common
// rows by their dispatch codes (three tests each), every other by op and class
template <class K, bool ABI, class V>
__device__ __forceinline__ void tile_row(const V &v, const Row16 &o, uint32_t plain, Cx<typename K::R> *acc) {
    const uint32_t code = ABI ? (uint32_t)R_OTHER : ((o.w.x | plain) & H_CODE);
    if (code < 4) {
        if (code < 2) {
            if (code == R_TENSOR_IMAG) tile_contribution<K, 4, C_IMAG, ABI>(v, o, acc);
            else tile_contribution<K, 6, C_IMAG, ABI>(v, o, acc);
        } else {
            if (code == R_WEDGE_ONE) tile_contribution<K, 5, C_ONE, ABI>(v, o, acc);
            else tile_closure_term<K, 4>(v, o, acc);
        }
    } else if (code < 8) {
        if (code < 6) {
            if (code == R_WEYL_A_REAL) tile_contribution<K, 2, C_REAL, ABI>(v, o, acc);
            else tile_contribution<K, 3, C_REAL, ABI>(v, o, acc);
        } else {
            if (code == R_PROP_IMAG) tile_vector_propagator<K>(v, o);
            else tile_closure_term<K, 2>(v, o, acc);
        }
    } else {
        Row16 q = o;
        q.w.x |= plain;
        const uint32_t op = o.op();
        if (!ABI && op == 7) tile_propagator<K, 7, ABI>(v, q);  // (in a batch the contributions here are rare)
        else if (!ABI && op == 8) tile_propagator<K, 8, ABI>(v, q);
        else if (op == 4) tile_contribution<K, 4, kClassOfRow, ABI>(v, q, acc);
        else if (op == 6) tile_contribution<K, 6, kClassOfRow, ABI>(v, q, acc);
        else if (op == 5) tile_contribution<K, 5, kClassOfRow, ABI>(v, q, acc);
        else if (op == 2) tile_contribution<K, 2, kClassOfRow, ABI>(v, q, acc);
        else if (op == 3) tile_contribution<K, 3, kClassOfRow, ABI>(v, q, acc);
        else if (op == 11) tile_closure<K>(v, q, acc);
        else if (op == 9) tile_propagator<K, 9, ABI>(v, q);
        else if (ABI && op == 7) tile_propagator<K, 7, ABI>(v, q);
        else if (ABI && op == 8) tile_propagator<K, 8, ABI>(v, q);
        else if (op == 10) tile_identity<K>(v, q);
        else if (op == kOpLoad) tile_load<K>(v, q, acc);
        else tile_clear<K>(v, q);
    }
}

// entry n of a folded table in the kind's values, from its list and the constants in the kind's layout
template <class K>
__device__ __forceinline__ Pair<typename K::R> fold_entry(const uint32_t *entries, uint32_t n, const typename K::Const *constants,
                                                          uint32_t scales, uint32_t factors) {
    typedef typename K::R R;
    typedef typename K::Const Const;
    const Const *sre = constants, *sim = sre + scales, *fre = sim + scales, *fim = fre + factors;
    const uint32_t kind = entries[2 * n] >> 28, a = entries[2 * n] & 0xfffffff, b = entries[2 * n + 1];
    Cx<R> x = kind == FOLD_SCALE_FACTOR ? cx(cast<R>(sre[a]), cast<R>(sim[a])) : cx(cast<R>(fre[a]), cast<R>(fim[a]));
    if (kind == FOLD_SCALE_FACTOR || kind == FOLD_FACTOR_FACTOR) x = x * cx(cast<R>(fre[b]), cast<R>(fim[b]));
    if (kind == FOLD_MINUS_I) x = x * cx(konst<R>(0.0), konst<R>(-1.0));
    Pair<R> o;
    o.re = x.re;
    o.im = x.im;
    return o;
}

// a plan's folded table (one thread per entry)
template <class K>
__global__ void fold_constants_kernel(const uint32_t *entries, uint32_t count, const typename K::Const *constants,
                                      uint32_t scales, uint32_t factors, Pair<typename K::R> *out) {
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < count) out[n] = fold_entry<K>(entries, n, constants, scales, factors);
}

// whether a reduced output is an infinity or a NaN
__device__ __forceinline__ bool not_finite(double x) {
    return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000;
}

// the levels of one item: level 0's sources, then each level's tasks in the lane order, a block
// barrier after each level (views of a compile-time point count address slots without products)
template <class K, bool ABI, class V>
__device__ __forceinline__ void run_levels(const V &v, const TiledPlan &p, double *forms64, uint32_t tl, bool active,
                                           uint32_t plain) {
    typedef typename K::R R;
    typedef typename K::Den Den;
    const uint32_t lanes = p.lanes, levels = p.levels;
    const uint4 *ins = p.ins;
    const uint32_t *order = p.order;
    for (uint32_t lv = 0; lv < levels; lv++) {
        const uint32_t j0 = __ldg(p.level_first + lv), j1 = active ? __ldg(p.level_first + lv + 1) : 0;
        if (lv == 0) {
            // the reciprocals of the propagators' norms, by the lanes the few sources leave idle
            R *recip = const_cast<R *>(v.rec_);
            for (uint32_t j = active ? lanes - 1 - tl : ~0u; j < p.recips; j += lanes) {
                const uint32_t f = __ldg(p.recip_forms + j);
                Den q[4];
                for (int c = 0; c < 4; c++) q[c] = narrow<Den>(forms64[v.at(f * 4 + c)]);
                recip[v.at(j)] = form_reciprocal<K>(q);
            }
            for (uint32_t j = j0 + tl; j < j1; j += lanes) {
                const uint32_t t = __ldg(order + j);
                // sources: f64 wavefunctions from the f64 forms and constants, narrowed
                Row16 o;
                for (const uint4 *at = ins + t; !(t & kNoTask); at++) {
                    o.w = __ldg(at);
                    double mom[4];
                    for (int c = 0; c < 4; c++) mom[c] = forms64[v.at(o.f0() * 4 + c)];
                    double fr = __ldg(p.f64 + o.x()), fi = __ldg(p.f64 + p.factors + o.x()), mass = __ldg(p.s64 + o.s());
                    W w[4];
                    int m = source_values(o.y(), mass, mom, w);
                    Cx<R> vals[4];
                    for (int c = 0; c < m; c++) {
                        double sr = fr * w[c].re - fi * w[c].im, si = fr * w[c].im + fi * w[c].re;
                        vals[c] = cx(narrow<R>(sr), narrow<R>(si));
                        v.put(o.a() + c, vals[c]);
                    }
                    if (o.w.x & H_WB) v.writeback(o.c(), vals, m);
                    if (o.w.x & H_END) break;
                }
            }
        } else {
            // Each lane runs its tasks, which end at an instruction of H_END. The next task's first
            // instruction is known while a task runs and the one after it is being fetched, so in
            // blocks of one point, where every lane fetches its own instructions and the points'
            // shared memory leaves L1 little room for them, the next task's first lines are
            // prefetched at once. (The order arrays end with two lane counts of padding and the
            // instructions with a line of it, so the fetches ahead need no bounds test.)
            uint32_t j = j0 + tl;
            uint32_t next_task = __ldg(order + j), task_after = __ldg(order + j + lanes);
            while (j < j1) {
                const uint32_t t = next_task;
                next_task = task_after;
                j += lanes;
                task_after = __ldg(order + j + lanes);
                if (t & kNoTask) continue;
                const uint4 *at = ins + t;
                Row16 o;
                uint4 next = __ldg(at);
                if (V::kPoints == 1) {
                    prefetch_l1(ins + (next_task & ~kNoTask));
                    prefetch_l1(ins + (next_task & ~kNoTask) + 7);
                }
                Cx<R> acc[6];
#pragma unroll
                for (int c = 0; c < 6; c++) acc[c] = cx(konst<R>(0.0), konst<R>(0.0));
                do {  // each next instruction is fetched while its predecessor runs
                    o.w = next;
                    next = __ldg(++at);
                    tile_row<K, ABI>(v, o, plain, acc);
                } while (!(o.w.x & H_END));
            }
        }
        __syncthreads();
        if (lv == 0 && !is_f64<Den>::value) {
            // the forms into df64 pairs, in place
            if (active)
                for (uint32_t q = tl; q < 4 * p.forms; q += lanes) {
                    uint32_t at = v.at(q);
                    reinterpret_cast<D *>(forms64)[at] = narrow<D>(forms64[at]);
                }
            __syncthreads();
        }
    }
}

// ABI: the C ABI's mode (arena in and out) or a batch's (outputs only). FAR: for launches with a plan of
// more entries than 16 bits index (rare, and a kernel of its own, since the index's upper half costs
// the others registers: df64 12 -> 24 bytes of spills, 65 537 points of the 3-jet mix 6.17 -> 6.29 ms)
template <class K, bool ABI, bool FAR = false>
__global__ void __launch_bounds__(512, 1) run_tiled(TiledLaunch L) {
    typedef typename K::R R;
    typedef typename K::Den Den;
    typedef typename K::Amp Amp;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned long long next_item[2];  // by turns: this item and (AHEAD) the one after it
    __shared__ uint32_t again;                   // (contracted) the item's points that are computed again, a bit each
    // The block's shared memory from its address in a register: taken from the array's symbol, every
    // row computes that address again (6 of 190 instructions; gg>ggg 4096 points 146 -> 143 us,
    // qg>qgg 125 -> 130 M points/s). The C ABI's kernel has no register left for it.
    unsigned char *block = smem;
    if (!ABI) {
        uint32_t window;
        asm volatile("mov.u32 %0, %1;" : "=r"(window) : "r"((uint32_t)__cvta_generic_to_shared(smem)));
        block = (unsigned char *)__cvta_shared_to_generic(window);
    }
    const unsigned long long total = L.item_first[L.nplans];
    // The counter's answer comes from L2. Asked for an item ahead, it comes while the item's forms wait
    // for memory: the df64 plans run one or two blocks per SM, whose other blocks do not cover that wait
    // (65 537 points of the 3-jet mix: 6.93 -> 6.14 ms). In f64 four blocks cover it, and one more value
    // that stays through the levels is spilled, to the little L1 that the instructions stream
    // through (4096 points of gg>ggg: 143 -> 153 us).
    constexpr bool AHEAD = !is_f64<R>::value;
    if (AHEAD) {
        if (threadIdx.x == 0) next_item[0] = atomicAdd(L.counter, 1ull);
        __syncthreads();
    }
    for (uint32_t turn = 0;; turn ^= AHEAD) {
        if (!AHEAD) {
            if (threadIdx.x == 0) next_item[0] = atomicAdd(L.counter, 1ull);
            __syncthreads();
        }
        const unsigned long long item = next_item[turn];
        if (item >= total) break;
        uint32_t k = 0;
        while (item >= L.item_first[k + 1]) k++;
        const TiledPlan &p = L.plans[k];
        const uint32_t np = p.points, lanes = p.lanes;
        if (ABI && threadIdx.x == 0) {
            abi_item.cre = L.cre;
            abi_item.cim = L.cim;
            abi_item.ld = L.ld;
            abi_item.first = (item - L.item_first[k]) * np;
            abi_item.count = L.count[k];
        }
        // this thread: lane tl of point pw; the threads of no group only meet the barriers
        const uint32_t groups = 32 / np, x = threadIdx.x & 31, q = x / np, pw = x - q * np;
        const uint32_t tl = (threadIdx.x >> 5) * groups + q;
        const bool active = q < groups;
        SlotView<K, ABI, 0, FAR> v;
        // forms, amplitudes, currents, terms, reciprocals: each region a multiple of the next one's
        // access size
        double *forms64 = (double *)(block + L.const_bytes);
        v.mom = (const Den *)forms64;
        v.amp_ = (Pair<Amp> *)(forms64 + (size_t)4 * p.forms * np);
        v.cur_ = (Pair<R> *)(v.amp_ + (size_t)p.amp_slots * np);
        v.term_ = (double *)(v.cur_ + (size_t)p.cur_slots * np);
        v.rec_ = (const R *)(v.term_ + (size_t)p.terms * np);
        const Pair<R> *near = (const Pair<R> *)block;
        v.folded_ = p.near == p.entries ? near : (const Pair<R> *)p.folded;
        for (uint32_t n = threadIdx.x; n < p.near; n += blockDim.x)
            ((Pair<R> *)block)[n] = ABI ? fold_entry<K>(p.entry_list, n, (const typename K::Const *)p.kconst, p.scales, p.factors)
                                       : ldg_pair((const Pair<R> *)p.folded + n);
        v.np = np;
        v.pw = pw;
        // a point whose outputs are not all finite is computed again with the plain formulas
        uint32_t plain = 0;
        while (true) {
            bool bad = false;
            unsigned long long ahead = 0;
            if (AHEAD && threadIdx.x == 0 && !plain) ahead = atomicAdd(L.counter, 1ull);
            if (active) {
                const uint32_t count = L.count[k];
                const size_t mine = (size_t)(item - L.item_first[k]) * np + pw;
                const size_t point = mine < count ? mine : count - 1;  // padding points redo the last point, unwritten
                // forms, f64: from the external momenta (0.0 + c0 p + c1 p + ..., in term order), or
                // the uploaded planes
                for (uint32_t q = tl; q < 4 * p.forms; q += lanes) {
                    uint32_t f = q >> 2, c = q & 3;
                    double val;
                    if (ABI && L.mom) {
                        val = L.mom[(size_t)q * L.ld + point];
                    } else {
                        uint32_t t0 = __ldg(p.form_terms + 2 * f), n = __ldg(p.form_terms + 2 * f + 1);
                        const double *ext = L.external[k];
                        val = 0.0;
                        for (uint32_t t = 0; t < n; t++) {
                            double term = __dmul_rn(__ldg(p.coefficients + t0 + t),
                                                    ext[((size_t)__ldg(p.term_slots + t0 + t) * 4 + c) * count + point]);
                            val = t == 0 ? __dadd_rn(0.0, term) : __dadd_rn(val, term);
                        }
                    }
                    forms64[q * np + pw] = val;
                }
                // the C ABI's mode: live-in currents and every amplitude from the global arena
                if (ABI) {
                    for (uint32_t j = 0; j < p.nloads; j++) {
                        uint32_t plane = __ldg(p.loads + 3 * j), slot = __ldg(p.loads + 3 * j + 1), n = __ldg(p.loads + 3 * j + 2);
                        for (uint32_t c = tl; c < n; c += lanes)
                            v.put(slot + c, cx(((const R *)L.cre)[(plane + c) * L.ld + point],
                                               ((const R *)L.cim)[(plane + c) * L.ld + point]));
                    }
                    for (uint32_t a = tl; a < p.amp_slots; a += lanes) {
                        uint32_t plane = __ldg(p.amp_planes + a);
                        v.put_amp(a, ((const Amp *)L.are)[plane * L.ld + point], ((const Amp *)L.aim)[plane * L.ld + point]);
                    }
                } else {
                    for (uint32_t a = tl; a < p.amp_slots; a += lanes) v.put_amp(a, konst<Amp>(0.0), konst<Amp>(0.0));
                    // a term whose amplitude no closure makes: the term of a zero amplitude
                    for (uint32_t t = tl; t < p.terms; t += lanes) v.put_term(t, konst<Amp>(0.0), konst<Amp>(0.0));
                }
            }
            if (AHEAD && threadIdx.x == 0 && !plain) next_item[turn ^ 1] = ahead;
            __syncthreads();  // the forms and live-in values are in
            // batches of one point per block (six-leg plans, gg>ggg) and of eight (the 5-leg quark
            // plans at two blocks per SM) run a copy of the levels with that count built in; in the C
            // ABI's kernel more copies of the levels cost registers
            const bool all_near = p.near == p.entries;
            if (!ABI && !FAR && np == 1 && all_near)
                run_levels<K, ABI>(v.template with_points<1>(near), p, forms64, tl, active, plain);
            else if (!ABI && !FAR && np == 8 && all_near)
                run_levels<K, ABI>(v.template with_points<8>(near), p, forms64, tl, active, plain);
            else
                run_levels<K, ABI>(v, p, forms64, tl, active, plain);
            if (ABI) {
                // (the point again from the item: nothing of it stays in registers through the levels)
                const unsigned long long at = abi_item.first + pw;
                if (active && at < abi_item.count)
                    for (uint32_t a = tl; a < p.amp_slots; a += lanes) {
                        uint32_t plane = __ldg(p.amp_planes + a);
                        Amp re, im;
                        v.amp(a, re, im);
                        ((Amp *)L.are)[plane * L.ld + at] = re;
                        ((Amp *)L.aim)[plane * L.ld + at] = im;
                    }
            } else if (active && (size_t)(item - L.item_first[k]) * np + pw < L.count[k] &&
                       (!K::contracted || !plain || again >> pw & 1)) {
                // the resolved reduction from zero: out[point][o] = 0 + w fma(re, re, im im) + ...
                const size_t point = (size_t)(item - L.item_first[k]) * np + pw;
                double *out = L.output[k] + point * p.outputs;
                for (uint32_t o = tl; p.terms && o < p.outputs; o += lanes) {
                    double acc = 0.0;
                    for (uint32_t j = __ldg(p.red_offsets + o), e = __ldg(p.red_offsets + o + 1); j < e; j++)
                        acc = __dadd_rn(acc, __dmul_rn(__ldg(p.red_weights + j), v.term_[v.at(j)]));
                    out[o] = acc;
                    bad |= not_finite(acc);
                }
                for (uint32_t o = tl; !p.terms && o < p.outputs; o += lanes) {
                    double acc = 0.0;
                    for (uint32_t j = __ldg(p.red_offsets + o), e = __ldg(p.red_offsets + o + 1); j < e; j++) {
                        uint32_t s = __ldg(p.red_slots + j);
                        double re = 0.0, im = 0.0;
                        if (s != ~0u) {
                            Amp ar, ai;
                            v.amp(s, ar, ai);
                            re = to_f64_value(ar);
                            im = to_f64_value(ai);
                        }
                        acc = __dadd_rn(acc, __dmul_rn(__ldg(p.red_weights + j), __fma_rn(re, re, __dmul_rn(im, im))));
                    }
                    out[o] = acc;
                    bad |= not_finite(acc);
                }
            }
            // (after this barrier the block's shared memory is free for the next item)
            if (ABI) {
                __syncthreads();
                break;
            }
            if (!__syncthreads_or(bad) || plain) break;
            // With contracted multiply-adds the plain formulas round otherwise: only those points' outputs are
            // replaced, so that a point's bits do not depend on the points beside it. (In the other kinds a
            // finite point gets the same bits again, and df64 has no registers to spare.)
            if (K::contracted) {
                if (threadIdx.x == 0) again = 0;
                __syncthreads();
                if (bad) atomicOr(&again, 1u << pw);
            }
            plain = H_PLAIN;
        }
    }
}

}  // namespace pacuda
