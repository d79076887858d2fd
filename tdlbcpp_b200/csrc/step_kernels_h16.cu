// 16-bit deviation storage (FP16 and BF16) instances of the step kernels
// (step_kernels.cuh). Populations are stored as f - w_d * rho0; collision and
// LES run in FP32. One, two and four cells per thread.
#include "step_kernels.cuh"

namespace tdlb {

static inline unsigned blocks16(long long n, int threads) { return (unsigned)((n + threads - 1) / threads); }

static inline unsigned grid16(const StepArgs& a, int V) {
    if (a.part == 2) return listed_blocks(a.zone.count, V);
    return blocks16(a.g.rows() * (a.g.jp / V), 128);
}

template <typename S, int V, bool LES, int PART>
static cudaError_t simple16_part(const StepArgs& a, cudaStream_t st) {
    return launch_step_kernel<kChained<PART>>(k_step_simple<S, V, LES, false, true, PART>, grid16(a, V), st, a.A, a.B, a.Nu, a.F, a.mask,
                                    a.g, a.p, launch_walk<k_step_simple<S, V, LES, false, true, PART>, true>(a));
}

template <typename S, int V, bool LES>
static cudaError_t simple16_les(const StepArgs& a, cudaStream_t st) {
    if (a.part == 1) return simple16_part<S, V, LES, 1>(a, st);
    if (a.part == 2) return simple16_part<S, V, LES, 2>(a, st);
    return simple16_part<S, V, LES, 0>(a, st);
}

template <typename S, int V>
static cudaError_t simple16(const StepArgs& a, cudaStream_t st) {
    return a.les ? simple16_les<S, V, true>(a, st) : simple16_les<S, V, false>(a, st);
}

template <typename S, int V, bool LES, int PART>
static cudaError_t eso16_part(const StepArgs& a, cudaStream_t st) {
    const unsigned grid = grid16(a, V);
    if (a.even)
        return launch_step_kernel<kChained<PART>>(k_step_esotwist<S, V, LES, false, true, true, PART>, grid, st, a.A, a.Nu, a.F, a.mask, a.g,
                                        a.p, launch_walk<k_step_esotwist<S, V, LES, false, true, true, PART>, true>(a));
    return launch_step_kernel<kChained<PART>>(k_step_esotwist<S, V, LES, false, true, false, PART>, grid, st, a.A, a.Nu, a.F, a.mask, a.g,
                                    a.p, launch_walk<k_step_esotwist<S, V, LES, false, true, false, PART>, true>(a));
}

template <typename S, int V, bool LES>
static cudaError_t eso16_les(const StepArgs& a, cudaStream_t st) {
    if (a.part == 1) return eso16_part<S, V, LES, 1>(a, st);
    if (a.part == 2) return eso16_part<S, V, LES, 2>(a, st);
    return eso16_part<S, V, LES, 0>(a, st);
}

template <typename S, int V>
static cudaError_t eso16(const StepArgs& a, cudaStream_t st) {
    return a.les ? eso16_les<S, V, true>(a, st) : eso16_les<S, V, false>(a, st);
}

cudaError_t launch_step_simple_h16(const StepArgs& a, cudaStream_t st) {
    if (!a.collide || a.from_moments) return cudaErrorInvalidValue;   // 16-bit state is always populations
    return with_storage(a.storage, [&](auto s) {
        using S = decltype(s);
        if constexpr (sizeof(S) == 4) return cudaErrorInvalidValue;
        else return a.vec == 1 ? simple16<S, 1>(a, st) : a.vec == 2 ? simple16<S, 2>(a, st) : simple16<S, 4>(a, st);
    });
}

cudaError_t launch_step_esotwist_h16(const StepArgs& a, cudaStream_t st) {
    if (!a.collide || a.from_moments) return cudaErrorInvalidValue;
    return with_storage(a.storage, [&](auto s) {
        using S = decltype(s);
        if constexpr (sizeof(S) == 4) return cudaErrorInvalidValue;
        else return a.vec == 1 ? eso16<S, 1>(a, st) : a.vec == 2 ? eso16<S, 2>(a, st) : eso16<S, 4>(a, st);
    });
}

template <typename S, bool SIMPLE, bool EVEN>
static cudaError_t box16(const StepArgs& a, cudaStream_t st) {
    return launch_step_kernel<true>(a.les ? k_box_step<S, SIMPLE, true, EVEN> : k_box_step<S, SIMPLE, false, EVEN>,
                                     blocks16(a.n_box, 128), st, a.A, a.B, a.Nu, a.F, a.mask, a.g, a.p, a.box_cells, a.n_box, a.rr, a.rw);
}

cudaError_t launch_box(const StepArgs& a, bool simple, cudaStream_t st) {
    if (!a.collide || a.from_moments || !a.rr.on() || !a.rw.on()) return cudaErrorInvalidValue;
    if (a.n_box <= 0) return cudaSuccess;
    return with_storage(a.storage, [&](auto s) {
        using S = decltype(s);
        if constexpr (sizeof(S) == 4) return cudaErrorInvalidValue;
        else {
            if (simple) return box16<S, true, true>(a, st);
            return a.even ? box16<S, false, true>(a, st) : box16<S, false, false>(a, st);
        }
    });
}

}  // namespace tdlb
