// Device side of the PK iteration shared by the vector passes (pcg.cu) and by
// the row passes that carry a step of the iteration in their loads and stores
// (op_impl.cuh): the scalar tails of the reductions and those loads and stores.
#pragma once

#include "fft_kernels.cuh"
#include "pk_state.hpp"
#include "reduce.cuh"

namespace asb {

// The gap buffers hold v = u + (g0 - gshift) uncentred after an evaluation;
// every later consumer centres on the fly with gc(), which is bit-identical to
// the reference's stored g = Real(v - Real(alpha)) (contact_solver.cpp:283-285),
// so centring costs no pass of its own.
template <typename T>
__device__ __forceinline__ T gc(T v, T aT) { return v - aT; }

// Scalar tail of the rsum / den pass (thread 0 of the last block).
// acc = {sum_C r, sum_C g t, sum_C r t, sum_C t};
// den = sum_C Real(r - rm) t, linear in rm: sum_C r t - rm sum_C t.
template <typename T>
__device__ inline void rden_tail(PkState* st, const double (&acc)[4]) {
    st->mv++;
    st->rsum = acc[0];
    st->num = acc[1];
    st->rmean = (double)(T)(st->nc ? acc[0] / st->nc : 0.0);
    const double den = acc[2] - st->rmean * acc[3], num = acc[1];
    st->den = den;
    if (den > 0.0 && isfinite(den) && isfinite(num)) {
        const T tau = (T)(num / den);
        st->tau = (double)tau;
        st->tau_ov = st->gg > 0.0 ? (double)(T)(num * num / (den * st->gg)) : (double)tau;
    } else {
        st->halt = H_IDENT;  // no usable direction: identification step
    }
}

// The pending load rescale of an instance (PkState::scale / scale_add),
// read once at kernel entry: the iterate is Real(x f) + a of the stored x
// (bit-identical to the reference's p(i) *= f, where a = 0).
template <typename T>
struct PScale {
    T f, a;
    __device__ explicit PScale(const PkState* st) : f((T)st->scale), a((T)st->scale_add) {}
    __device__ __forceinline__ T operator()(T x) const { return x * f + a; }
};

// Scalar tail of evaluate() (thread 0 of the last block); final_mode: of the
// returned iterate (k_eval), without the loop's decisions.
// acc = {sum_C v, n_C, min v, sum p v, sum p}
template <typename T>
__device__ inline void eval_tail(const PkParams& P, PkState* st, const double (&acc)[5],
                                 bool final_mode) {
    if (!final_mode) {
        if (!st->u_fresh) st->mv++;
        st->u_fresh = 0;
        st->pk_due = 1;
    }
    const int nc = (int)acc[1];
    const double alpha = nc ? acc[0] / nc : acc[2];
    const double gmin = acc[2] - alpha;
    const double aT = (double)(T)alpha, gmT = (double)(T)gmin;
    const double gcs = acc[0] - (double)nc * aT;
    st->nc = nc;
    st->gsum = acc[0];
    st->vmin = acc[2];
    st->par ^= 1;
    st->mask_stale = 0;
    st->alpha_prev = st->alpha;
    st->alpha = alpha;
    st->gmin = gmin;
    double ar = alpha, gr = gmin;
    if (nc > 0) {  // refine_contact_mean (contact_solver.cpp:94-99)
        const double d = gcs / nc;
        ar += d;
        gr -= d;
    }
    const double PG = P.P_total * P.g_ref;
    const double G = acc[3] - (aT + gmT) * acc[4];
    st->alpha_ref = ar;
    st->gmin_ref = gr;
    st->pv = acc[3];
    st->gcs = gcs;
    st->G = G;
    st->fw = G / PG;
    st->pen = fmax(0.0, -gr) / P.g_ref;
    st->psum = acc[4];
    st->load = fabs(acc[4] - P.P_total) / P.P_total;
    st->finite = isfinite(acc[0]) && isfinite(acc[2]) && isfinite(acc[4]) && isfinite(acc[3]);
    if (final_mode) return;
    if (!st->finite) {
        st->status = ST_NONFINITE;
        st->halt = H_FINAL;
        return;
    }
    if (st->load <= P.load_tol && st->fw <= P.tol && st->pen <= P.tol) {
        st->status = ST_CONVERGED;
        st->u_fresh = 1;
        st->halt = H_FINAL;
        return;
    }
    const double merit = fmax(st->fw, st->pen);
    if (P.keep_best && merit < st->best_merit) {
        st->best_merit = merit;
        st->copy_best = 1;
    }
    if (merit < st->seen_merit * (1.0 - 1e-4)) {
        st->seen_merit = merit;
        st->stall = 0;
    } else if (++st->stall >= P.stall_limit) {
        st->halt = H_STALL;
        return;
    }
    if (nc < 2) st->halt = H_IDENT;
}

// ---- steps of the iteration in the row passes ------------------------------------
// A pass of its own for each of them re-read (and the apply before it wrote) a
// whole field and cost a launch and a reduction's tail.  B200, a solve's
// iteration with separate passes / so: FP64 free-space 128 40.6 / 38.0 us,
// 768-sided 95.0 / 90.0, FP32-FP64 mixed 1024 88.3 / 79.8, six 2048 solves 266
// / 257 ms.  u's store and load and r's store are saved at any contact.
// Each works on the pairs of cells (2n, 2n + 1) of a row that its thread
// transforms, n = t + m TT: first the mask of all of them (no contact, no
// traffic), then the fields, those of U pairs in flight together: a warp in
// contact otherwise waits for one load after another.  begin() reads the
// instance's scalars once.  Per launch in a free-space solve at Ns = 2048, one
// pair after the other / so: FP32 evaluate 39.0 / 35.5 us, line sums 32.6 /
// 29.2, direction 21.8 / 18.9; FP64 fields 53.4 / 45.9, 36.9 / 31.7, 21.8 / 20.0.

// the largest power of two up to `most` that divides nv
__host__ __device__ constexpr int pairs_in_flight(int nv, int most) {
    int u = most;
    while (nv % u) u /= 2;
    return u;
}

// The direction update t = chi_C(z_f + beta t) in the forward row load of the
// t apply (t is 0 off contact: k_pupd clears what leaves it).
template <typename T, typename Z>
struct LoadDirection {
    using Real = T;
    static constexpr bool kBatch = true;
    const PkParams* P;
    const PkState* st;
    const T* z;
    const T* ga;
    const T* gb;
    T* t;
    const uint8_t* mask;
    int pitch;
    long bs;
    // of the instance
    const T* g = nullptr;
    T zm = T(0), beta = T(0), aT = T(0);
    bool pre = false;
    __device__ __forceinline__ void begin() {
        const PkState* sb = st + blockIdx.y;
        g = sb->par ? gb : ga;
        zm = (T)sb->zmean;
        beta = (T)sb->beta;
        aT = (T)sb->alpha;
        pre = P[blockIdx.y].precond != 0;
    }
    template <int NV, int TT, int RPT>
    __device__ __forceinline__ void all(int row, int t0, cplx<Z> (&v)[RPT]) const {
        const size_t i0 = blockIdx.y * bs + (size_t)row * pitch + 2 * t0;
        uchar2 m[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k)
            m[k] = *reinterpret_cast<const uchar2*>(mask + i0 + 2 * k * TT);
        // f = z - zmean, or the centred gap: the same subtraction
        const T* src = pre ? z : g;
        const T c = pre ? zm : aT;
        constexpr int U = pairs_in_flight(NV, sizeof(T) == 8 ? 4 : 8);
#pragma unroll
        for (int k0 = 0; k0 < NV; k0 += U) {
            cplx<T> d[U], f[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const size_t i = i0 + 2 * (k0 + k) * TT;
                d[k] = f[k] = mk<T>(T(0), T(0));
                if (m[k0 + k].x | m[k0 + k].y) {
                    d[k] = *reinterpret_cast<const cplx<T>*>(t + i);
                    f[k] = *reinterpret_cast<const cplx<T>*>(src + i);
                }
            }
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const uchar2 mm = m[k0 + k];
                const cplx<T> e = mk<T>(mm.x ? (T)((T)(f[k].x - c) + beta * d[k].x) : T(0),
                                        mm.y ? (T)((T)(f[k].y - c) + beta * d[k].y) : T(0));
                if (mm.x | mm.y)
                    *reinterpret_cast<cplx<T>*>(t + i0 + 2 * (k0 + k) * TT) = e;
                v[k0 + k] = mk<Z>((Z)e.x, (Z)e.y);
            }
        }
    }
};

// evaluate() in the inverse row store of the p apply (the sums of k_eval; u
// itself is not stored).  u0 (defect-corrected applies): u = u0 + z.
template <typename T, typename Z>
struct StoreEval {
    using Real = T;
    static constexpr bool kFinish = true;
    static constexpr int kPartials = 5;
    static constexpr bool kBatch = true;
    const PkParams* P;
    PkState* st;
    const T* u0;
    const T* g0;
    const T* p;
    T* ga;
    T* gb;
    uint8_t* mask;
    double* part;
    int pitch;
    long bs;
    // sum_C v, n_C, min v, pv, psum
    double acc[kPartials] = {0.0, 0.0, (double)INFINITY, 0.0, 0.0};
    T* g = nullptr;
    T gs = T(0), f = T(0), a = T(0);
    bool stale = false;
    __device__ __forceinline__ void begin() {
        const PkState* sb = st + blockIdx.y;
        g = sb->par ? ga : gb;
        stale = sb->mask_stale != 0;
        gs = (T)P[blockIdx.y].gshift;
        f = (T)sb->scale;
        a = (T)sb->scale_add;
    }
    template <int NV, int TT, int RPT>
    __device__ __forceinline__ void all(int row, int t0, const cplx<Z> (&v)[RPT], uint32_t mb) {
        const size_t i0 = blockIdx.y * bs + (size_t)row * pitch + 2 * t0;
        constexpr int U = pairs_in_flight(NV, 4);
#pragma unroll
        for (int k0 = 0; k0 < NV; k0 += U) {
            cplx<T> h[U], w[U], q[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const size_t i = i0 + 2 * (k0 + k) * TT;
                h[k] = *reinterpret_cast<const cplx<T>*>(g0 + i);
                if (u0) w[k] = *reinterpret_cast<const cplx<T>*>(u0 + i);
                q[k] = mk<T>(T(0), T(0));
                if (stale || pair_mask(mb, k0 + k)) q[k] = *reinterpret_cast<const cplx<T>*>(p + i);
            }
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const size_t i = i0 + 2 * (k0 + k) * TT;
                T ux = (T)v[k0 + k].x, uy = (T)v[k0 + k].y;
                if (u0) {
                    ux = w[k].x + ux;
                    uy = w[k].y + uy;
                }
                const T vx = ux + (h[k].x - gs), vy = uy + (h[k].y - gs);
                *reinterpret_cast<cplx<T>*>(g + i) = mk<T>(vx, vy);
                acc[2] = fmin(acc[2], fmin((double)vx, (double)vy));
                T px = T(0), py = T(0);
                const uint32_t m = pair_mask(mb, k0 + k);
                if (stale || m) {
                    px = q[k].x * f + a;
                    py = q[k].y * f + a;
                    const uint32_t mn = (px > T(0) ? 1u : 0u) | (py > T(0) ? 2u : 0u);
                    if (px > T(0)) { acc[0] += (double)vx; acc[1] += 1.0; }
                    if (py > T(0)) { acc[0] += (double)vy; acc[1] += 1.0; }
                    if (stale || mn != m)
                        *reinterpret_cast<uint16_t*>(mask + i) = (uint16_t)((mn & 1u) | (mn & 2u) << 7);
                }
                acc[3] += (double)px * (double)vx;
                acc[3] += (double)py * (double)vy;
                acc[4] += (double)px + (double)py;
            }
        }
    }
    __device__ void finish(double*) {
        PkState* sb = st + blockIdx.y;
        const int kinds[kPartials] = {0, 0, 1, 0, 0};
        if (grid_reduce_last<kPartials>(acc, kinds, part + (size_t)blockIdx.y * kPartStride,
                                &sb->counter[0]) && threadIdx.x == 0)
            eval_tail<T>(P[blockIdx.y], sb, acc, false);
    }
};

// The line-search sums in the inverse row store of the t apply (r itself is
// not stored).
template <typename T, typename Z>
struct StoreLineSums {
    using Real = T;
    static constexpr bool kFinish = true;
    static constexpr int kPartials = 4;
    static constexpr bool kBatch = true;
    PkState* st;
    const T* ga;
    const T* gb;
    const T* t;
    const uint8_t* mask;
    double* part;
    int pitch;
    long bs;
    double acc[kPartials] = {0.0, 0.0, 0.0, 0.0};  // sum_C r, sum_C g t, sum_C r t, sum_C t
    const T* g = nullptr;
    T aT = T(0);
    __device__ __forceinline__ void begin() {
        const PkState* sb = st + blockIdx.y;
        g = sb->par ? gb : ga;
        aT = (T)sb->alpha;
    }
    template <int NV, int TT, int RPT>
    __device__ __forceinline__ void all(int row, int t0, const cplx<Z> (&v)[RPT], uint32_t mb) {
        if (!mb) return;
        const size_t i0 = blockIdx.y * bs + (size_t)row * pitch + 2 * t0;
        constexpr int U = pairs_in_flight(NV, 4);
#pragma unroll
        for (int k0 = 0; k0 < NV; k0 += U) {
            cplx<T> d[U], h[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const size_t i = i0 + 2 * (k0 + k) * TT;
                d[k] = h[k] = mk<T>(T(0), T(0));
                if (pair_mask(mb, k0 + k)) {
                    d[k] = *reinterpret_cast<const cplx<T>*>(t + i);
                    h[k] = *reinterpret_cast<const cplx<T>*>(g + i);
                }
            }
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const uint32_t m = pair_mask(mb, k0 + k);
                if (m & 1u) add((T)v[k0 + k].x, h[k].x, d[k].x);
                if (m & 2u) add((T)v[k0 + k].y, h[k].y, d[k].y);
            }
        }
    }
    __device__ __forceinline__ void add(T r, T h, T d) {
        const double td = (double)d;
        acc[0] += (double)r;
        acc[1] += (double)gc(h, aT) * td;
        acc[2] += (double)r * td;
        acc[3] += td;
    }
    __device__ void finish(double*) {
        PkState* sb = st + blockIdx.y;
        const int kinds[kPartials] = {0, 0, 0, 0};
        if (grid_reduce_last<kPartials>(acc, kinds, part + (size_t)blockIdx.y * kPartStride,
                                &sb->counter[4]) && threadIdx.x == 0)
            rden_tail<T>(sb, acc);
    }
};

// The fields of a PK iteration of gridDim.y instances, as the row passes see
// them (instances N apart).
template <typename T>
struct PkFields {
    const PkParams* P;
    PkState* st;
    const T* g0;
    T* p;
    T* t;
    const T* z;
    T* ga;
    T* gb;
    uint8_t* mask;
    double* part;
    // defect-corrected applies (FP64 fields, FP32 transforms): p0 and u0 = S p0
    const T* p0;
    const T* u0;
};

// The two applies of a PK iteration of B instances with the iteration's steps
// in their row passes: eval: u = S p and evaluate(); else the direction
// update t, r = S t and the line-search sums.  Gated by each instance's halt.
// defect: FP64 fields, transforms in FP32 (u = u0 + S_32(p - p0), r = S_32 t).
struct Operator;
void pk_apply(Operator& op, const PkFields<float>& f, bool eval, bool defect, void* spec,
              cudaStream_t s, int B);
void pk_apply(Operator& op, const PkFields<double>& f, bool eval, bool defect, void* spec,
              cudaStream_t s, int B);

}  // namespace asb
