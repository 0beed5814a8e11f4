// Host helpers of the on-chip executor (tiled_host.h).
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <memory>
#include <vector>

#include "../../include/pacman_recurrence.h"
#include "../../include/pacuda_b200.h"
#include "tiled.cuh"
#include "tiled_host.h"

namespace pacuda {

namespace {

// The arrays of a device plan, in one allocation and one copy (several of each were a few percent of a
// small plan's first call).
struct Slab {
    struct Array {
        void **dst;
        const void *src;
        size_t at, bytes;
    };
    std::vector<Array> arrays;
    size_t total = 0;
    // room for `n` values that *dst is to point at, filled from `src` where there is one
    template <class T> void add(T **dst, const T *src, size_t n) {
        arrays.push_back({(void **)dst, src, total, src ? n * sizeof(T) : 0});
        total += (std::max<size_t>(1, n) * sizeof(T) + 255) / 256 * 256;
    }
    template <class T> void add(T **dst, const std::vector<T> &v) { add(dst, v.data(), v.size()); }
    // (waits for the copy)
    bool upload(void **slab, cudaStream_t s) {
        if (cudaMalloc(slab, total) != cudaSuccess) {
            *slab = nullptr;
            return false;
        }
        std::unique_ptr<uint8_t[]> host(new uint8_t[total]);
        size_t end = 0;
        for (const Array &a : arrays) {
            *a.dst = (uint8_t *)*slab + a.at;
            if (a.bytes) memcpy(host.get() + a.at, a.src, a.bytes);
            if (a.bytes) end = a.at + a.bytes;
        }
        return cudaMemcpyAsync(*slab, host.get(), end, cudaMemcpyHostToDevice, s) == cudaSuccess &&
               cudaStreamSynchronize(s) == cudaSuccess;
    }
};

}  // namespace

// the f64 kind with contracted multiply-adds (tiled_fma.cu, compiled with -fmad=true)
const void *tiled_fma_kernel(bool abi, bool far);
// the other kinds' kernels for tables of more entries than 16 bits index (tiled_far.cu)
const void *tiled_far_kernel(int kernel, bool abi);
void tiled_fma_fold(const uint32_t *entries, uint32_t count, const void *constants, uint32_t scales, uint32_t factors,
                    void *out, cudaStream_t s);

namespace {

template <class K> const void *kernel_of(bool abi) {
    return abi ? (const void *)run_tiled<K, true> : (const void *)run_tiled<K, false>;
}

const void *kernel_for(int kernel, bool abi = false, bool far = false) {
    if (far && kernel != PACUDA_B200_KERNEL_F64_FMA) return tiled_far_kernel(kernel, abi);
    switch (kernel) {
    case PACMAN_RECURRENCE_KERNEL_F64: return kernel_of<KindF64>(abi);
    case PACUDA_B200_KERNEL_F64_FMA: return tiled_fma_kernel(abi, far);
    case PACMAN_RECURRENCE_KERNEL_MIXED: return kernel_of<KindMixed>(abi);
    case PACMAN_RECURRENCE_KERNEL_MIXED64: return kernel_of<KindMixed64>(abi);
    default: return kernel_of<KindDF64>(abi);
    }
}
}  // namespace

void TiledDevice::release() {
    cudaFree(slab);
    slab = nullptr;
    ins = bare = nullptr;
    loads = amp_planes = orders = level_firsts = entries = recip_forms = nullptr;
    folded = nullptr;
    ok = false;
}

bool pack_ins(const Ins &i, bool end, uint4 &w) {
    // (a closure's f records its global amplitude plane for the host; the executor reads its slot)
    uint32_t f = ins_kind(i) == K_CLOSURE ? 0 : i.f, f0 = f & 0xffff, f1 = f >> 16;
    uint32_t a = i.a, b = i.b, c = i.c, s = i.s, x = i.x, y = i.y;
    auto split = [](uint32_t &low, uint32_t &high) {  // an entry's index (Row16 entry_s, _x, _y)
        high = low >> 16;
        low &= 0xffff;
    };
    if (ins_kind(i) == K_CONTRIB && ins_op(i) != kOpLoad) split(s, x);
    else if (ins_kind(i) == K_PROP || ins_kind(i) == K_IDENTITY) split(x, c);
    else if (ins_kind(i) == K_CLOSURE) split(y, x);
    for (uint32_t field : {a, b, c, s, x, y})
        if (field > 0xffff) return false;
    if (ins_count(i) > C_GENERAL || f0 > 255 || f1 > 255) return false;
    const uint32_t flags = ins_flags(i);
    const bool contribution = ins_kind(i) == K_CONTRIB && ins_op(i) != kOpLoad, last = !contribution || (flags & F_LAST);
    uint32_t head = row_code(i) | ins_count(i) << 4 | ins_op(i) << 8;
    if (end) head |= H_END;
    if (contribution && last && !(flags & F_NOSTORE)) head |= H_STORE;
    if (flags & F_ACC0) head |= H_ACC0;
    if (flags & F_TERM) head |= H_TERM;
    if (contribution && (flags & F_FIRST) && (flags & F_INIT)) head |= H_SET;
    if (last && (flags & F_WB)) head |= H_WB;
    w.x = head | f0 << 16 | f1 << 24;
    w.y = a | b << 16;
    w.z = c | s << 16;
    w.w = x | y << 16;
    return true;
}

bool upload_schedule(TiledDevice &t, int threads, const TiledConstants &c, cudaStream_t s) {
    Folds folds;
    fold_constants(t.host, c.scale_re, c.scale_im, c.factor_re, c.factor_im, folds);
    t.entry_count = (uint32_t)folds.entries.size() / 2;
    t.recips = (uint32_t)folds.reciprocals.size();
    std::vector<uint8_t> end(folds.ins.size(), 0);
    for (size_t k = 1; k < folds.task_first.size(); k++) end[folds.task_first[k] - 1] = 1;
    std::vector<uint4> packed(folds.ins.size()), bare(folds.ins.size());
    for (size_t n = 0; n < packed.size(); n++) {
        Ins i = folds.ins[n];
        bool ok = pack_ins(i, end[n], packed[n]);
        if (ins_kind(i) == K_PROP) i.s = kNoReciprocal;
        if (!ok || !pack_ins(i, end[n], bare[n])) {
            t.host.why = "an instruction's field does not fit the on-chip executor's 16-byte form";
            t.ok = false;
            return false;
        }
    }
    // fetched (not run) ahead of a task's end, and beside the positions without a task
    const uint32_t padding = (uint32_t)packed.size();
    packed.resize(packed.size() + 8, make_uint4(0, 0, 0, 0));
    bare.resize(packed.size(), make_uint4(0, 0, 0, 0));
    t.levels = (uint32_t)t.host.level_first.size() - 1;
    t.threads = threads;
    std::vector<uint32_t> first, firsts;
    // one order per distinct lane count: blocks of b per SM with P points give
    // tiled_lanes(P, tiled_block_threads(threads, b)) lanes, and many pairs give the same count
    std::vector<bool> made(kMaxLanes + 1, false);
    for (int b : kBlockChoices)
        for (uint32_t np = 1; threads > 0 && np <= kMaxPoints; np++) {
            uint32_t lanes = tiled_lanes(np, tiled_block_threads(threads, b));
            if (lanes == 0 || lanes > kMaxLanes || made[lanes]) continue;
            made[lanes] = true;
            std::vector<uint32_t> order, lf;
            lane_order(t.host, lanes, order, lf);
            // each position holds its task's first instruction
            t.order_at[lanes] = first.size();
            t.level_at[lanes] = firsts.size();
            for (uint32_t task : order) first.push_back(task == ~0u ? kNoTask | padding : folds.task_first[task]);
            firsts.insert(firsts.end(), lf.begin(), lf.end());
        }
    // the executor fetches two positions of a lane ahead: up to two lane counts past the last one
    first.insert(first.end(), 3 * kMaxLanes, kNoTask | padding);
    Slab slab;
    slab.add(&t.ins, packed);
    slab.add(&t.orders, first);
    slab.add(&t.level_firsts, firsts);
    slab.add(&t.loads, t.host.loads);
    slab.add(&t.amp_planes, t.host.amp_planes);
    slab.add(&t.entries, folds.entries);
    slab.add(&t.recip_forms, folds.reciprocals);
    slab.add(&t.bare, bare);
    slab.add((uint4 **)&t.folded, (const uint4 *)nullptr, t.entry_count);  // (16 bytes an entry)
    t.ok = threads > 0 && slab.upload(&t.slab, s);
    return t.ok;
}

bool fold_values(const TiledDevice &t, int kernel, const void *constants, uint32_t scales, uint32_t factors,
                 cudaStream_t s) {
    if (!t.entry_count) return true;
    auto fold = [&](auto k) {
        typedef decltype(k) K;
        fold_constants_kernel<K><<<(t.entry_count + 127) / 128, 128, 0, s>>>(
            t.entries, t.entry_count, (const typename K::Const *)constants, scales, factors, (Pair<typename K::R> *)t.folded);
    };
    switch (kernel) {
    case PACMAN_RECURRENCE_KERNEL_F64: fold(KindF64()); break;
    case PACUDA_B200_KERNEL_F64_FMA: tiled_fma_fold(t.entries, t.entry_count, constants, scales, factors, t.folded, s); break;
    case PACMAN_RECURRENCE_KERNEL_MIXED: fold(KindMixed()); break;
    case PACMAN_RECURRENCE_KERNEL_MIXED64: fold(KindMixed64()); break;
    default: fold(KindDF64()); break;
    }
    return cudaGetLastError() == cudaSuccess;
}

size_t tiled_point_bytes(const TiledDevice &t, uint32_t forms, int kernel, bool keep) {
    const Schedule &s = t.host;
    const size_t recips = keep ? t.recips : 0;
    size_t value = kernel == PACMAN_RECURRENCE_KERNEL_MIXED || kernel == PACMAN_RECURRENCE_KERNEL_MIXED64 ? 4 : 8;
    size_t per_point = 2 * value * s.cur_slots + 2 * 8 * s.amp_slots + 8 * (s.terms + recips) + 8 * 4 * (size_t)forms;
    return (per_point + 15) / 16 * 16;
}

int tiled_threads(int kernel, int blocks) {
    cudaFuncAttributes attr, abi;
    if (cudaFuncGetAttributes(&attr, kernel_for(kernel, false)) != cudaSuccess ||
        cudaFuncGetAttributes(&abi, kernel_for(kernel, true)) != cudaSuccess)
        return 0;
    attr.numRegs = std::max(attr.numRegs, abi.numRegs);
    attr.maxThreadsPerBlock = std::min(attr.maxThreadsPerBlock, abi.maxThreadsPerBlock);
    int dev = 0, regs = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&regs, cudaDevAttrMaxRegistersPerBlock, dev);
    int per_warp = ((attr.numRegs * 32 + 255) / 256) * 256;
    int warps = per_warp ? regs / per_warp : 16;
    warps = std::min(warps, attr.maxThreadsPerBlock / 32);
    warps = std::max(1, std::min(warps, 16));
    return tiled_block_threads(32 * warps, blocks);
}

size_t tiled_max_smem(int kernel, int blocks) {
    cudaFuncAttributes attr, abi;
    if (cudaFuncGetAttributes(&attr, kernel_for(kernel, false)) != cudaSuccess ||
        cudaFuncGetAttributes(&abi, kernel_for(kernel, true)) != cudaSuccess)
        return 0;
    attr.sharedSizeBytes = std::max(attr.sharedSizeBytes, abi.sharedSizeBytes);
    int dev = 0, smem = 0, per_sm = 0, reserved = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    // with several blocks per SM each gets its share of the SM's shared memory
    size_t limit = blocks > 1 ? std::min<size_t>(smem, (size_t)(per_sm - blocks * reserved) / blocks) : (size_t)smem;
    return limit > attr.sharedSizeBytes ? limit - attr.sharedSizeBytes : 0;
}

int tiled_auto_blocks(int kernel, const PlanSize &size) {
    PlanSize plan = size;
    plan.points = 0;
    std::vector<PlanShape> shape;
    size_t table = 0;
    auto fits = [&](int blocks) {
        return launch_shapes({plan}, tiled_threads(kernel, blocks), tiled_max_smem(kernel, blocks), false, table, shape);
    };
    uint32_t one = fits(1) ? shape[0].points : 0;
    // the choices to try, most blocks first
    static const int few[] = {4, 2};
    const int *first = one && one <= 4 ? few : few + 1;
    for (const int *b = first; b != few + 2; b++)
        if (fits(*b)) return *b;
    return 1;
}

void describe(const TiledDevice &t, uint32_t forms, const PlanShape &shape, size_t point_bytes, size_t const_bytes,
              TiledPlan &p, int blocks) {
    p.ins = shape.keep ? t.ins : t.bare;
    const uint32_t lanes = tiled_lanes(shape.points, tiled_block_threads(t.threads, blocks));
    p.order = t.orders + t.order_at[lanes];
    p.level_first = t.level_firsts + t.level_at[lanes];
    p.levels = t.levels;
    p.cur_slots = t.host.cur_slots;
    p.amp_slots = t.host.amp_slots;
    p.terms = t.host.terms;
    p.forms = forms;
    p.points = shape.points;
    p.lanes = lanes;
    p.point_bytes = (uint32_t)point_bytes;
    p.loads = t.loads;
    p.nloads = (uint32_t)t.host.loads.size() / 3;
    p.amp_planes = t.amp_planes;
    p.folded = t.folded;
    p.entries = t.entry_count;
    p.near = 16 * (size_t)t.entry_count <= const_bytes ? t.entry_count : 0;
    p.recip_forms = t.recip_forms;
    p.recips = shape.keep ? t.recips : 0;
}

bool launch_tiled(int kernel, const TiledLaunch &args, int threads, size_t smem, int grid, cudaStream_t stream) {
    const void *fn = kernel_for(kernel, args.abi, args.far);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return false;
    void *params[] = {(void *)&args};
    return cudaLaunchKernel(fn, dim3(grid), dim3(threads), params, smem, stream) == cudaSuccess;
}

}  // namespace pacuda
