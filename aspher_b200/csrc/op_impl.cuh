// The per-size implementations of the operators: the three passes of the
// free-space and the periodic apply and of the full-grid |k| preconditioner,
// as templates over the compute grid.  Their kernels are compiled by
// op_free_*.cu and op_periodic_*.cu (one translation unit per pipeline and
// precision, the PK steps apart); operators.cu uses the layout constants alone.
#pragma once

#include "fft_kernels.cuh"
#include "fft_launch.cuh"
#include "functors.cuh"
#include "ops.hpp"
#include "pk_device.cuh"
#include "reduce.cuh"

namespace asb {

// the two launches of the split column transform (variant 0 only): parity 0
// writes its half to acc, parity 1 adds it and writes the column in place
template <typename T, int LH, int NCM1, class Mult>
void launch_col_split(cplx<T>* spec, cplx<T>* acc, int nrows, int ndata, Mult m,
                      cudaStream_t s, const int* gate, int B = 1) {
    constexpr int V = vclamp(LH, 0);
    constexpr int ct = col_ct_v<T>(LH, NCM1, V), thr = col_threads<T>(LH, NCM1, V);
    constexpr int sm = col_smem<T>(LH, ct);
    const dim3 grid(NCM1 / ct + 1, B);
    auto go = [&](auto all) {
        auto k0 = col_split_kernel<T, LH, NCM1, V, 0, decltype(all)::value, Mult>;
        auto k1 = col_split_kernel<T, LH, NCM1, V, 1, decltype(all)::value, Mult>;
        fft_attrs((const void*)k0, sm);
        fft_attrs((const void*)k1, sm);
        launch_pdl(k0, grid, thr, sm, s, spec, acc, nrows, ndata, m, tw<T>(LH), tw<T>(2 * LH),
                   gate);
        launch_pdl(k1, grid, thr, sm, s, spec, acc, nrows, ndata, m, tw<T>(LH), tw<T>(2 * LH),
                   gate);
    };
    if (ndata >= LH) go(std::true_type{});
    else go(std::false_type{});
}

#define ASB_V_SWITCH(VV, L, ...)                                                   \
    switch (VV) {                                                                  \
        case 0: { constexpr int V = vclamp(L, 0); __VA_ARGS__; } break;            \
        case 1: { constexpr int V = vclamp(L, 1); __VA_ARGS__; } break;            \
        case 2: { constexpr int V = vclamp(L, 2); __VA_ARGS__; } break;            \
        case 3: { constexpr int V = vclamp(L, 3); __VA_ARGS__; } break;            \
        default: throw Error(-1, "FFT launch variant out of range");              \
    }

// ONLY >= 0: launch variant ONLY whatever v is (one instantiation per pass:
// the grids above kMaxVariantNs)
template <typename T, int LR, bool PAD, int ONLY = -1, class Load, class Store>
void row_fwd_v(int v, Load ld, Store st, int nrows, cudaStream_t s, const int* gate, int B) {
    if constexpr (ONLY >= 0) {
        launch_row_fwd<T, LR, PAD, ONLY, Load, Store>(ld, st, nrows, s, gate, B);
    } else {
        ASB_V_SWITCH(v, LR, (launch_row_fwd<T, LR, PAD, V, Load, Store>(ld, st, nrows, s, gate, B)));
    }
}
template <typename T, int LR, bool PAD, int ONLY = -1, class Load, class Store>
void row_inv_v(int v, Load ld, Store st, int nrows, cudaStream_t s, const int* gate, int B) {
    if constexpr (ONLY >= 0) {
        launch_row_inv<T, LR, PAD, ONLY, Load, Store>(ld, st, nrows, s, gate, B);
    } else {
        ASB_V_SWITCH(v, LR, (launch_row_inv<T, LR, PAD, V, Load, Store>(ld, st, nrows, s, gate, B)));
    }
}
template <typename T, int LC, int NCM1, bool PAD, int ONLY = -1, class Mult>
void col_v(int v, cplx<T>* spec, int nrows, int ndata, Mult m, cudaStream_t s, const int* gate,
           int B) {
    if constexpr (ONLY >= 0) {
        launch_col<T, LC, NCM1, PAD, ONLY, Mult>(spec, nrows, ndata, m, s, gate, B);
    } else {
        ASB_V_SWITCH(v, LC, (launch_col<T, LC, NCM1, PAD, V, Mult>(spec, nrows, ndata, m, s, gate, B)));
    }
}
// tile width of column variant v (runtime view of the constexpr table)
template <typename T, int LC, int NCM1>
int col_ct_rt(int v) {
    int ct = 1;
    ASB_V_SWITCH(v, LC, ct = col_ct_v<T>(LC, NCM1, V));
    return ct;
}

// ----------------------------------------------------------------------------
// per-size implementation
// ----------------------------------------------------------------------------
template <typename T, int NS>
struct FreeImpl {
    static constexpr int LR = NS, LC = 2 * NS;
    // the length-2Ns column in one CTA's shared memory (all sizes but FP64
    // at Ns = 8192); otherwise the column pass runs as two length-Ns halves
    // (col_split_kernel), instantiated for Ns >= kSplitMin
    static constexpr bool kFits = col_fits<T>(LC);
    static constexpr bool kSplitOK = NS >= kSplitMin && NS % 3 != 0 && col_fits<T>(LR);
    // rows and columns in one CTA each (every size but FP64 above 8192)
    static constexpr bool kSupported = row_smem_v<T>(LR, 0) <= kSmemPerSM && (kFits || kSplitOK);
    static constexpr bool kAllV = NS <= kMaxVariantNs;
    // the one launch variant of the grids above kMaxVariantNs
    static constexpr VariantRow kDefault = default_variants(OP_FFT, sizeof(T) == 8, NS);
    static constexpr int kRV = vclamp(LR, kDefault.rv), kCV = vclamp(LC, kDefault.cv);
    static constexpr int kOnlyR = kAllV ? -1 : kRV, kOnlyC = kAllV ? -1 : kCV;
    static bool split(const Operator& op) { return !kFits || (kSplitOK && op.split_cols); }
    // spectrum sized for the widest tile (16 columns); the split form keeps
    // its first half-column result in a second spectrum-shaped block after
    // the B instances' spectra
    static size_t spec_elems(bool sp) { return (size_t)(LR + 16) * NS * (sp ? 2 : 1); }
    static int ct(int cv, bool sp) {
        if (sp) return col_ct_v<T>(LR, LR, vclamp(LR, 0));
        return kAllV ? col_ct_rt<T, LC, LR>(cv) : col_ct_v<T>(LC, LR, kCV);
    }

    // row_fwd(ld) -> col(x Kh) -> row_inv(st); ld / st see the Ns x Ns
    // field(s), of which the first op.Nl rows hold data (all of them unless
    // the operator is embedded): the row passes run on those rows alone and
    // the column pass takes the rest as zero.
    template <class Load, class Store>
    static void apply(const Operator& op, Load ld, Store st, cplx<T>* spec, cudaStream_t s,
                      const int* gate, int B, const T* kh_over = nullptr) {
        if constexpr (!kSupported) {
            throw Error(-1, "free-space FP64 apply above grid_size 8192 is not supported (its "
                            "rows and half columns do not fit one CTA's shared memory); use FP32");
        } else {
            const int dbl = sizeof(T) == 8;
            const int rv = op.rowv[dbl], cv = op.colv[dbl], c = op.ct[dbl];
            const T* kh = kh_over ? kh_over : (dbl ? (const T*)op.kh_d : (const T*)op.kh_f);
            const long bsp = (long)(LR / c + 1) * NS * c;
            const int nd = op.Nl;
            row_fwd_v<T, LR, true, kOnlyR>(rv, ld, StoreTiled<T>{spec, NS, c, bsp}, nd, s, gate, B);
            if (split(op)) {
                if constexpr (kSplitOK)
                    launch_col_split<T, LR, LR>(spec, spec + (size_t)B * bsp, NS, nd,
                                                KhMult<T>{kh, NS + 1, LC, c}, s, gate, B);
            } else {
                if constexpr (kFits)
                    col_v<T, LC, LR, true, kOnlyC>(cv, spec, NS, nd, KhMult<T>{kh, NS + 1, LC, c},
                                                  s, gate, B);
            }
            row_inv_v<T, LR, true, kOnlyR>(rv, LoadTiled<T>{spec, NS, c, bsp}, st, nd, s, gate, B);
            count_launches(split(op) ? 4 : 3);
            ASB_CUDA(cudaGetLastError());
        }
    }

    static void matvec(const Operator& op, const T* x, T* y, cplx<T>* spec, cudaStream_t s,
                       const int* gate, int B) {
        const long bx = (long)NS * NS;
        apply(op, LoadRealRows<T>{x, NS, bx}, StoreRealRows<T>{y, NS, bx}, spec, s, gate, B);
    }

    // an apply with a step of the PK iteration in its store (and load)
    template <class Load, class Store>
    static void pk(const Operator& op, Load ld, Store st, cplx<T>* spec, cudaStream_t s,
                   const int* gate, int B) {
        apply(op, ld, st, spec, s, gate, B);
    }

    // an embedded operator's apply on the caller's own layout
    static void apply_block(const Operator& op, const T* x, T* y, long nl, cplx<T>* spec,
                            cudaStream_t s) {
        apply(op, LoadBlockRows<T>{x, op.Nl, nl}, StoreBlockRows<T>{y, op.Nl, nl}, spec, s,
              nullptr, 1);
    }
};

// The two applies of a PK iteration on the impl's operator: evaluate() in the
// row store of the p apply, the direction update and the line-search sums in
// the row load and store of the t apply.  F: the solver's precision, T: the transform's.
template <class Impl, typename F, typename T>
void pk_eval_apply(const Operator& op, const PkFields<F>& f, cplx<T>* spec, cudaStream_t s, int B) {
    const int Ns = op.Ns;
    const long bx = (long)Ns * Ns;
    const StoreEval<F, T> st{f.P, f.st, f.u0, f.g0, f.p, f.ga, f.gb, f.mask, f.part, Ns, bx};
    if constexpr (sizeof(F) != sizeof(T))
        Impl::pk(op, LoadDiffRows{f.p, f.p0, Ns, bx, f.st}, st, spec, s, &f.st->halt, B);
    else
        Impl::pk(op, LoadRealRows<T>{f.p, Ns, bx, f.st}, st, spec, s, &f.st->halt, B);
}
template <class Impl, typename F, typename T>
void pk_line_apply(const Operator& op, const PkFields<F>& f, cplx<T>* spec, cudaStream_t s, int B) {
    const int Ns = op.Ns;
    const long bx = (long)Ns * Ns;
    Impl::pk(op, LoadDirection<F, T>{f.P, f.st, f.z, f.ga, f.gb, f.t, f.mask, Ns, bx},
             StoreLineSums<F, T>{f.st, f.ga, f.gb, f.t, f.mask, f.part, Ns, bx}, spec, s,
             &f.st->halt, B);
}

template <typename T, int NS>
struct PeriodicImpl {
    static constexpr int LR = NS / 2, LC = NS;
    // rows and columns in one CTA each (every size but FP64 above 8192)
    static constexpr bool kSupported = row_smem_v<T>(LR, 0) <= kSmemPerSM && col_fits<T>(LC);
    static constexpr bool kAllV = NS <= kMaxVariantNs;
    static size_t spec_elems() { return (size_t)(LR + 16) * NS; }
    static int ct(int cv) {
        return kAllV ? col_ct_rt<T, LC, LR>(cv)
                     : col_ct_v<T>(LC, LR, vclamp(LC, default_variants(OP_PERIODIC, sizeof(T) == 8, NS).cv));
    }

    static constexpr VariantRow kDefault = default_variants(OP_PERIODIC, sizeof(T) == 8, NS);
    static constexpr int kRV = vclamp(LR, kDefault.rv), kCV = vclamp(LC, kDefault.cv);
    static constexpr int kOnlyR = kAllV ? -1 : kRV, kOnlyC = kAllV ? -1 : kCV;

    template <class Load, class Mult, class Store>
    static void apply(int rv, int cv, Load ld, Mult mult, Store st, cplx<T>* spec, cudaStream_t s,
                      const int* gate, int B) {
        if constexpr (!kSupported) {
            throw Error(-1, "periodic FP64 apply above grid_size 8192 is not supported (its "
                            "column does not fit one CTA's shared memory); use FP32");
        } else {
            const int c = ct(cv);
            const long bsp = (long)(LR / c + 1) * NS * c;
            row_fwd_v<T, LR, false, kOnlyR>(rv, ld, StoreTiled<T>{spec, NS, c, bsp}, NS, s, gate, B);
            col_v<T, LC, LR, false, kOnlyC>(cv, spec, NS, NS, mult, s, gate, B);
            row_inv_v<T, LR, false, kOnlyR>(rv, LoadTiled<T>{spec, NS, c, bsp}, st, NS, s, gate, B);
            count_launches(3);
            ASB_CUDA(cudaGetLastError());
        }
    }

    // the multiplier scale / |m| from the operator's table of this precision
    // (the values PeriodicMult forms per element, one load instead of an
    // FP64 square root and division)
    static KhMult<T> mult(const Operator& op) {
        const int dbl = sizeof(T) == 8;
        const T* tab = dbl ? (const T*)(const void*)op.psym_d : (const T*)(const void*)op.psym_f;
        return KhMult<T>{tab, NS / 2 + 1, NS, op.ct[dbl]};
    }

    static void matvec(const Operator& op, const T* x, T* y, cplx<T>* spec, cudaStream_t s,
                       const int* gate, int B) {
        const int dbl = sizeof(T) == 8;
        const long bx = (long)NS * NS;
        apply(op.rowv[dbl], op.colv[dbl], LoadRealRows<T>{x, NS, bx}, mult(op),
              StoreRealRows<T>{y, NS, bx}, spec, s, gate, B);
    }

    template <class Load, class Store>
    static void pk(const Operator& op, Load ld, Store st, cplx<T>* spec, cudaStream_t s,
                   const int* gate, int B) {
        const int dbl = sizeof(T) == 8;
        apply(op.rowv[dbl], op.colv[dbl], ld, mult(op), st, spec, s, gate, B);
    }
};

// ----------------------------------------------------------------------------
// full-grid |k| preconditioner (reference: src/fourier_precond.cpp:12-116)
// ----------------------------------------------------------------------------
template <typename T>
struct LoadMaskCentered {  // contact ? g - T(gsum/ng) : 0, pairwise; g = v - T(alpha)
    const T* ga;  // the gap is in ga or gb (PkState::par)
    const T* gb;
    const uint8_t* mask;
    const PkState* st;
    int pitch;
    long bs;  // batch stride (elements); instance blockIdx.y uses st[blockIdx.y]
    __device__ __forceinline__ cplx<T> operator()(int row, int n) const {
        const PkState* sb = st + blockIdx.y;
        const int nc = sb->nc;
        const T gm = nc ? (T)(sb->gcs / nc) : T(0);
        // the solve loop keeps g uncentred (centred by Real(alpha) on the fly;
        // alpha is 0 for the standalone preconditioner)
        const T aT = (T)sb->alpha;
        const size_t i = blockIdx.y * bs + (size_t)row * pitch + 2 * n;
        const cplx<T> v = *reinterpret_cast<const cplx<T>*>((sb->par ? gb : ga) + i);
        const uchar2 m = *reinterpret_cast<const uchar2*>(mask + i);
        return mk<T>(m.x ? (T)((T)(v.x - aT) - gm) : T(0), m.y ? (T)((T)(v.y - aT) - gm) : T(0));
    }
};

template <typename T>
struct FourierMult {  // |k| / Ns^2 as the reference's float table, cast to T
    int Ns;
    float norm;
    __device__ __forceinline__ cplx<T> operator()(cplx<T> X, int kx, int ky) const {
        const int kof = ky < Ns / 2 ? ky : ky - Ns;
        const float w = (kx == 0 && ky == 0) ? 0.0f : norm * hypotf((float)kx, (float)kof);
        return cscale(X, (T)w);
    }
};

template <typename T>
struct StoreGather {  // z = contact ? G : 0; contact sum of G -> zmean
    T* z;
    const uint8_t* mask;
    int pitch;
    PkState* st;
    double* part;
    long bs;  // batch stride (elements); instance blockIdx.y uses st / part of its own
    static constexpr bool kFinish = true;
    static constexpr int kPartials = 1;
    double zs;
    __device__ __forceinline__ void operator()(int row, int n, cplx<T> v) {
        const size_t i = blockIdx.y * bs + (size_t)row * pitch + 2 * n;
        const uchar2 m = *reinterpret_cast<const uchar2*>(mask + i);
        *reinterpret_cast<cplx<T>*>(z + i) = mk<T>(m.x ? v.x : T(0), m.y ? v.y : T(0));
        if (m.x) zs += (double)v.x;
        if (m.y) zs += (double)v.y;
    }
    __device__ void finish(double*) {
        double a[kPartials] = {zs};
        const int kinds[kPartials] = {0};
        PkState* sb = st + blockIdx.y;
        double* pb = part + (size_t)blockIdx.y * kPartStride;
        if (grid_reduce_last<kPartials>(a, kinds, pb, &sb->counter[11]) && threadIdx.x == 0) {
            const int nc = sb->nc;
            sb->zmean = nc ? (double)(T)(a[0] / nc) : 0.0;
            sb->pc++;
        }
    }
};

template <typename T, int NS>
struct FourierImpl {
    using PI = PeriodicImpl<T, NS>;
    static void run(Operator& op, const T* ga, const T* gb, const uint8_t* mask, PkState* st,
                        T* z,
                    double* part, cudaStream_t s, const int* gate, int B, void* spec_b) {
        cplx<T>* spec = static_cast<cplx<T>*>(spec_b ? spec_b : op.spectrum(sizeof(T) == 8, s));
        int rv = 0, cv = 0;
        tuned_variants(OP_PERIODIC, sizeof(T) == 8, NS, rv, cv);
        const float norm = 1.0f / ((float)NS * (float)NS);
        const long bx = (long)NS * NS;
        PI::apply(rv, cv, LoadMaskCentered<T>{ga, gb, mask, st, NS, bx}, FourierMult<T>{NS, norm},
                  StoreGather<T>{z, mask, NS, st, part, bx, 0.0}, spec, s, gate, B);
    }
};

// the full-grid |k| preconditioner of an embedded grid: the masked centred
// residual convolved with the symbol's real-space kernel on the Nl torus by
// the compute grid's padded pipeline, gathered on contact with its contact
// sum (the same load and store as the periodic form)
template <typename T, int NS>
struct EmbeddedFourierImpl {
    static void run(Operator& op, const T* ga, const T* gb, const uint8_t* mask, PkState* st,
                        T* z,
                    double* part, cudaStream_t s, const int* gate, int B, void* spec_b) {
        if (!op.khp_canon)
            throw Error(-1, "fourier-fft preconditioner spectrum not built (set-up order)");
        cplx<T>* spec = static_cast<cplx<T>*>(spec_b ? spec_b : op.spectrum(sizeof(T) == 8, s));
        const long bx = (long)NS * NS;
        const T* kh = sizeof(T) == 8 ? (const T*)op.khp_d : (const T*)op.khp_f;
        FreeImpl<T, NS>::apply(op, LoadMaskCentered<T>{ga, gb, mask, st, NS, bx},
                               StoreGather<T>{z, mask, NS, st, part, bx, 0.0}, spec, s, gate, B,
                               kh);
    }
};

// ----------------------------------------------------------------------------
// size dispatch
// ----------------------------------------------------------------------------
#define ASB_SIZE_SWITCH(NSV, ...)                      \
    switch (NSV) {                                      \
        case 16: { constexpr int NS = 16; __VA_ARGS__; } break;     \
        case 32: { constexpr int NS = 32; __VA_ARGS__; } break;     \
        case 64: { constexpr int NS = 64; __VA_ARGS__; } break;     \
        case 128: { constexpr int NS = 128; __VA_ARGS__; } break;   \
        case 256: { constexpr int NS = 256; __VA_ARGS__; } break;   \
        case 512: { constexpr int NS = 512; __VA_ARGS__; } break;   \
        case 1024: { constexpr int NS = 1024; __VA_ARGS__; } break; \
        case 2048: { constexpr int NS = 2048; __VA_ARGS__; } break; \
        case 4096: { constexpr int NS = 4096; __VA_ARGS__; } break; \
        case 8192: { constexpr int NS = 8192; __VA_ARGS__; } break; \
        case 16384: { constexpr int NS = 16384; __VA_ARGS__; } break; \
        default: throw Error(-1, "grid_size must be a power of two in [16, 16384]"); \
    }
// the same with the embedded grids' sides of 3 2^k (free-space pipeline)
#define ASB_FREE_SWITCH(NSV, ...)                       \
    switch (NSV) {                                       \
        case 768: { constexpr int NS = 768; __VA_ARGS__; } break;   \
        case 1536: { constexpr int NS = 1536; __VA_ARGS__; } break; \
        case 3072: { constexpr int NS = 3072; __VA_ARGS__; } break; \
        default: ASB_SIZE_SWITCH(NSV, __VA_ARGS__)       \
    }

// what op_free_*.cu and op_periodic_*.cu define for their pipeline and T
// (F: the solver's precision of a PK step)
template <typename F, typename T>
void free_pk_eval(const Operator& op, const PkFields<F>& f, cplx<T>* spec, cudaStream_t s, int B);
template <typename F, typename T>
void free_pk_line(const Operator& op, const PkFields<F>& f, cplx<T>* spec, cudaStream_t s, int B);
template <typename F, typename T>
void periodic_pk_eval(const Operator& op, const PkFields<F>& f, cplx<T>* spec, cudaStream_t s,
                      int B);
template <typename F, typename T>
void periodic_pk_line(const Operator& op, const PkFields<F>& f, cplx<T>* spec, cudaStream_t s,
                      int B);
template <typename T>
void free_matvec(const Operator& op, const T* x, T* y, cplx<T>* spec, cudaStream_t s,
                 const int* gate, int B);
template <typename T>
void free_apply_block(const Operator& op, const T* x, T* y, cplx<T>* spec, cudaStream_t s);
template <typename T>
void embedded_precond(Operator& op, const T* ga, const T* gb, const uint8_t* mask, PkState* st,
                        T* z,
                      double* part, cudaStream_t s, const int* gate, int B, void* spec);
template <typename T>
void periodic_matvec(const Operator& op, const T* x, T* y, cplx<T>* spec, cudaStream_t s,
                     const int* gate, int B);
template <typename T>
void periodic_precond(Operator& op, const T* ga, const T* gb, const uint8_t* mask, PkState* st,
                        T* z,
                      double* part, cudaStream_t s, const int* gate, int B, void* spec);

}  // namespace asb
