// Host-side launchers of the FFT pass kernels (fft_kernels.cuh): launch
// shape of variant V, dynamic shared memory (with the opt-in attribute set
// once per kernel and device), persistent grids for the staged forms, and
// gridDim.y = B instances.  Shared by the operators' translation units.
#pragma once

#include "fft_kernels.cuh"
#include "ops.hpp"
#include "reduce.cuh"

#include <type_traits>
#include <utility>

namespace asb {

// small transforms run the small-CTA variant; those of 3 2^k points have two
// shapes, variant 2 and the other three
__host__ __device__ constexpr int vclamp(int L, int V) {
    return L % 3 == 0 ? (V == 2 ? 2 : 0) : (L >= 128 ? V : 3);
}

// the set-up's row passes: variant 0 but for rows of 16 points, which it would
// run in CTAs of 16 threads, half a warp of the reduction in their stores
__host__ __device__ constexpr int build_variant(int L) { return L < 32 ? 3 : 0; }

// Fastest (row, column) variant pairs measured on B200: every pair set on
// one operator (aspher_op_set_variants) and 6-20 of its applies timed in a
// CUDA graph (sides of 3 2^k: the passes alone); sizes not listed use variant
// 0.  Operator::autotune repeats the search in-process.
struct VariantRow {
    int kind, dbl, Ns, rv, cv;
};
constexpr VariantRow kVariantTable[] = {
    {0, 0, 64, 3, 3}, {0, 0, 128, 3, 3}, {0, 0, 256, 3, 3}, {0, 0, 512, 2, 1},
    {0, 0, 768, 2, 2}, {0, 0, 1024, 1, 2}, {0, 0, 1536, 0, 2}, {0, 0, 2048, 1, 2},
    {0, 0, 3072, 0, 0}, {0, 0, 4096, 0, 2}, {0, 0, 8192, 0, 0}, {0, 1, 64, 3, 3},
    {0, 1, 128, 3, 3}, {0, 1, 256, 3, 3}, {0, 1, 512, 3, 1}, {0, 1, 768, 2, 2},
    {0, 1, 1024, 1, 1}, {0, 1, 1536, 0, 2}, {0, 1, 2048, 1, 1}, {0, 1, 3072, 0, 0},
    {0, 1, 4096, 0, 2}, {1, 0, 128, 3, 3}, {1, 0, 256, 3, 3}, {1, 0, 512, 3, 3},
    {1, 0, 1024, 3, 1}, {1, 0, 2048, 2, 2}, {1, 0, 4096, 1, 2}, {1, 0, 8192, 0, 2},
    {1, 1, 128, 3, 3}, {1, 1, 256, 3, 3}, {1, 1, 512, 3, 3}, {1, 1, 1024, 3, 1},
    {1, 1, 2048, 2, 1}, {1, 1, 4096, 3, 0}, {1, 1, 8192, 0, 2},
};
constexpr VariantRow default_variants(int kind, int dbl, int Ns) {
    for (const VariantRow& e : kVariantTable)
        if (e.kind == kind && e.dbl == dbl && e.Ns == Ns) return e;
    return VariantRow{kind, dbl, Ns, 0, 0};
}

// max dynamic shared memory + max-shared carveout, once per kernel per device
void fft_attrs(const void* func, int bytes);
// CTAs of a persistent pass kernel: at most occupancy x SMs, at most `units`
int persistent_blocks(const void* func, int threads, int smem, int units);

// Launch of a pass kernel as a programmatic dependent of the kernel in front
// of it on the stream (the kernel begins with pdl_wait()).  On B200 an
// ordinary launch behind a running kernel starts on a grid of 2.05 us after
// its end (3.6-4.1 us per kernel for kernels of 0-2.3 us back to back on a
// stream, 1.9-2.5 us so; 16 and 592 CTAs), and a boundary between the kernel
// nodes of a graph costs 0.2 us less.
template <class... P, class... A>
void launch_pdl(void (*k)(P...), dim3 grid, int threads, int smem, cudaStream_t s, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    ASB_CUDA(cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...));
}

// values that a reducing store of a row pass writes per CTA to the instance's
// partials (Store::kPartials), 0 for the others
template <class S, class = void>
struct store_partials : std::integral_constant<int, 0> {};
template <class S>
struct store_partials<S, std::enable_if_t<(S::kPartials > 0)>>
    : std::integral_constant<int, S::kPartials> {};

// B > 1: gridDim.y = B instances (functors / gates / spectrum per instance)
template <typename T, int LR, bool PAD, int V, class Load, class Store>
void launch_row_fwd(Load ld, Store st, int nrows, cudaStream_t s, const int* gate, int B = 1) {
    constexpr int rb = row_rb_v<T>(LR, V), thr = row_threads<T>(LR, V);
    constexpr int sm = row_smem_v<T>(LR, V);
    static_assert(!Store::kFinish || thr % 32 == 0, "a reduction needs whole warps");
    auto k = row_fwd_kernel<T, LR, PAD, V, Load, Store>;
    fft_attrs((const void*)k, sm);
    const int gx = (nrows + rb - 1) / rb;
    launch_pdl(k, dim3(gx, B), thr, sm, s, ld, st, nrows, tw<T>(LR), tw<T>(2 * LR), gate);
}
template <typename T, int LR, bool PAD, int V, class Load, class Store>
void launch_row_inv(Load ld, Store st, int nrows, cudaStream_t s, const int* gate, int B = 1) {
    constexpr int rb = row_rb_v<T>(LR, V), thr = row_threads<T>(LR, V);
    constexpr int sm = row_smem_v<T>(LR, V);
    constexpr long rows = PAD ? LR : 2 * LR;  // of the whole grid
    static_assert(Store::kFinish == (store_partials<Store>::value > 0) &&
                      (rows + rb - 1) / rb * store_partials<Store>::value <= kPartStride,
                  "a reducing row pass writes past its instance's partials");
    static_assert(!Store::kFinish || thr % 32 == 0, "a reduction needs whole warps");
    auto k = row_inv_kernel<T, LR, PAD, V, Load, Store>;
    fft_attrs((const void*)k, sm);
    const int gx = (nrows + rb - 1) / rb;
    launch_pdl(k, dim3(gx, B), thr, sm, s, ld, st, nrows, tw<T>(LR), tw<T>(2 * LR), gate);
}
template <typename T, int LC, int NCM1, bool PAD, int V, class Mult>
void launch_col(cplx<T>* spec, int nrows, int ndata, Mult m, cudaStream_t s, const int* gate, int B = 1) {
    constexpr int ct = col_ct_v<T>(LC, NCM1, V), thr = col_threads<T>(LC, NCM1, V);
    constexpr int sm = col_smem_total<T, LC, NCM1, PAD, V>();
    auto k = col_kernel<T, LC, NCM1, PAD, V, Mult>;
    fft_attrs((const void*)k, sm);
    const int gx = col_staged<T, LC, NCM1, PAD, V>()
                       ? persistent_blocks((const void*)k, thr, sm, NCM1 / ct + 1)
                       : NCM1 / ct + 1;
    launch_pdl(k, dim3(gx, B), thr, sm, s, spec, nrows, ndata, m, tw<T>(LC), gate);
}


}  // namespace asb
