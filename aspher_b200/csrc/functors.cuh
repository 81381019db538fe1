// Load / store / multiplier functors of the row and column kernels shared by
// the operators (operators.cu) and the allocation-free entry point.
#pragma once

#include "fft_kernels.cuh"

namespace asb {

// Every functor offsets by blockIdx.y * bs (elements): instance blockIdx.y
// of a batched launch (bs = 0 or gridDim.y = 1 for a single field).
// The PK loop's pressure with the pending load rescale of instance
// blockIdx.y (PkState::scale / scale_add): Real(x f) + a.  Plain loads: the
// kernel in front writes the state, and a read-only load need not stay behind
// pdl_wait().
template <typename T>
__device__ __forceinline__ T pending_scale(const PkState* sc, T x) {
    const PkState* sb = sc + blockIdx.y;
    return x * (T)sb->scale + (T)sb->scale_add;
}

template <typename T>
struct LoadRealRows {  // z[n] = (x[row*pitch + 2n], x[row*pitch + 2n + 1])
    const T* x;
    int pitch;
    long bs;
    // optional: x is the PK loop's pressure, scaled by the pending load
    // rescale of sc[blockIdx.y] as it is loaded
    const PkState* sc = nullptr;
    __device__ __forceinline__ cplx<T> fix(cplx<T> v) const {
        if (sc) {
            v.x = pending_scale(sc, v.x);
            v.y = pending_scale(sc, v.y);
        }
        return v;
    }
    __device__ __forceinline__ cplx<T> operator()(int row, int n) const {
        return fix(*reinterpret_cast<const cplx<T>*>(x + blockIdx.y * bs + (size_t)row * pitch +
                                                      2 * n));
    }
};

template <typename T>
struct StoreRealRows {
    T* y;
    int pitch;
    long bs;
    static constexpr bool kFinish = false;
    __device__ __forceinline__ void operator()(int row, int n, cplx<T> z) const {
        *reinterpret_cast<cplx<T>*>(y + blockIdx.y * bs + (size_t)row * pitch + 2 * n) = z;
    }
    __device__ void finish(double*) const {}
};

// An embedded operator's caller field (Nl rows of Nl values): z[n] of the
// compute grid's row, 0 outside the caller's block.  Scalar accesses: an odd
// Nl leaves the rows at every alignment.
template <typename T>
struct LoadBlockRows {
    const T* x;
    int Nl;
    long bs;
    __device__ __forceinline__ cplx<T> operator()(int row, int n) const {
        cplx<T> z = mk<T>(T(0), T(0));
        if (row < Nl) {
            const T* r = x + blockIdx.y * bs + (size_t)row * Nl;
            if (2 * n < Nl) z.x = r[2 * n];
            if (2 * n + 1 < Nl) z.y = r[2 * n + 1];
        }
        return z;
    }
};

template <typename T>
struct StoreBlockRows {
    T* y;
    int Nl;
    long bs;
    static constexpr bool kFinish = false;
    __device__ __forceinline__ void operator()(int row, int n, cplx<T> z) const {
        if (row >= Nl) return;
        T* r = y + blockIdx.y * bs + (size_t)row * Nl;
        if (2 * n < Nl) r[2 * n] = z.x;
        if (2 * n + 1 < Nl) r[2 * n + 1] = z.y;
    }
    __device__ void finish(double*) const {}
};

// FP64 rows in, FP32 pairs out: x - x0, rounded once.  A defect-corrected FP64
// apply (pk_apply) transforms this difference in FP32.
struct LoadDiffRows {
    const double* x;
    const double* x0;
    int pitch;
    long bs;
    // optional: x is the PK loop's pressure with a pending load rescale
    // (see LoadRealRows)
    const PkState* sc = nullptr;
    __device__ __forceinline__ cplx<float> operator()(int row, int n) const {
        const size_t i = blockIdx.y * bs + (size_t)row * pitch + 2 * n;
        double2 v = *reinterpret_cast<const double2*>(x + i);
        if (sc) {
            v.x = pending_scale(sc, v.x);
            v.y = pending_scale(sc, v.y);
        }
        const double2 w = *reinterpret_cast<const double2*>(x0 + i);
        v.x -= w.x;
        v.y -= w.y;
        return mk<float>((float)v.x, (float)v.y);
    }
};

// the tiled half spectrum of row_fwd_kernel's stores and row_inv_kernel's loads
template <typename T>
struct StoreTiled {
    cplx<T>* base;
    int nrows, ct;
    long bs;
    static constexpr bool kFinish = false;
    static constexpr bool kTiled = true;
    __device__ void finish(double*) const {}
};

template <typename T>
struct LoadTiled {
    const cplx<T>* base;
    int nrows, ct;
    long bs;
};

// Free-space multiplier: real Kh, even-folded in ky, tiled like the spectrum
// with ct columns per tile and Ns+1 rows.
template <typename T>
struct KhMult {
    const T* kh;
    int nk;  // Ns + 1 rows
    int M;   // padded length 2 Ns
    int ct;
    __device__ __forceinline__ cplx<T> operator()(cplx<T> X, int kx, int ky) const {
        const int kf = ky <= (M >> 1) ? ky : M - ky;
        const T w = __ldg(&kh[(size_t)(kx / ct) * nk * ct + (size_t)kf * ct + (kx % ct)]);
        return cscale(X, w);
    }
};

// Periodic multiplier: scale / |m| in FP64, cast to T (periodic_fft_operator.cpp:34-47).
template <typename T>
struct PeriodicMult {
    double scale;
    int Ns;
    __device__ __forceinline__ cplx<T> operator()(cplx<T> X, int kx, int ky) const {
        const int my = ky < (Ns + 1) / 2 ? ky : ky - Ns;
        const double m2 = (double)kx * kx + (double)my * my;
        const T w = m2 > 0.0 ? (T)(scale / sqrt(m2)) : T(0);
        return cscale(X, w);
    }
};

}  // namespace asb
