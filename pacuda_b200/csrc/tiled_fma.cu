// The on-chip executor in f64 with multiply-adds contracted (PACUDA_B200_KERNEL_F64_FMA): the
// same source as the f64 kind, compiled in this file with -fmad=true, so that the compiler fuses
// a product and the sum it feeds into one DFMA (one rounding instead of two). Its values differ
// from the reference's f64 arithmetic in the last bits (about 1e-15 relative per operation); the
// plan's structure, order of operations and everything else are the f64 kind's.
#include "tiled.cuh"

namespace pacuda {

// a kind of its own (so that its kernels are not the -fmad=false f64 kind's instantiations)
struct KindF64Fma : Kind<double, double, double, double> {
    static constexpr bool contracted = true;
};

const void *tiled_fma_kernel(bool abi, bool far) {
    if (far) return abi ? (const void *)run_tiled<KindF64Fma, true, true> : (const void *)run_tiled<KindF64Fma, false, true>;
    return abi ? (const void *)run_tiled<KindF64Fma, true> : (const void *)run_tiled<KindF64Fma, false>;
}

void tiled_fma_fold(const uint32_t *entries, uint32_t count, const void *constants, uint32_t scales, uint32_t factors,
                    void *out, cudaStream_t s) {
    fold_constants_kernel<KindF64Fma><<<(count + 127) / 128, 128, 0, s>>>(entries, count, (const double *)constants,
                                                                          scales, factors, (Pair<double> *)out);
}

}  // namespace pacuda
