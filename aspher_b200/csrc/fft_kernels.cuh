// Row and column pass kernels of the 2-D real transforms.
//
// A 2-D r2c/c2r pair over an (nrows x 2*LR) real grid is split as:
//   row_fwd : per row, the real FFT of length 2*LR via a length-LR complex
//             FFT of z[n] = x[2n] + i x[2n+1] and the usual split step,
//             producing the LR+1 half-spectrum columns;
//   col     : per column, forward FFT of length LC, pointwise multiplier,
//             inverse FFT (fused: the spectrum never leaves the CTA);
//   row_inv : per row, the inverse split step and a length-LR complex FFT.
// PAD=true is the zero-padded (Hockney) case of the free-space operator:
// rows hold Ns real values padded to 2*Ns (so half of z is zero and those
// registers are never loaded), and columns hold Ns values padded to LC=2*Ns
// of which only the first Ns outputs are kept.
//
// The half spectrum lives in HBM in a column-tiled layout:
//   elem(row, k) = base[(k / ct) * nrows * ct + row * ct + (k % ct)]
// so a column CTA streams one contiguous tile and a row CTA of RB rows
// touches RB*ct contiguous elements per tile.
//
// Batched solves launch every kernel with gridDim.y = instances; the load /
// store functors offset their pointers by blockIdx.y times a batch stride,
// and instance b's spectrum is the b-th block of gridDim.x column tiles.
//
// Launch shapes are variants (V = 0..kVariants-1) trading registers per
// thread (RPT elements, radix <= RPT), CTA size and CTAs per SM; the
// operator picks one row variant and one column variant per size and
// precision (a default table, or the autotuner in operators.cu).
#pragma once

#include <type_traits>

#include "fft_block.cuh"
#include "pk_state.hpp"

namespace asb {

constexpr int kVariants = 4;
// Batched launches (gridDim.y = instances) read instance b's gate at
// gate[b * kGateStride]: the gates live in consecutive PkState records, which
// the kernel in front and a reducing store write (hence no __restrict__).
constexpr int kGateStride = (int)(sizeof(PkState) / sizeof(int));
static_assert(sizeof(PkState) % sizeof(int) == 0, "PkState must be a whole number of ints");
constexpr int kSmemPerSM = 227 * 1024;

// ---- variant tables -----------------------------------------------------------------
// (points per thread, threads per CTA, CTAs per SM), measured on B200 over
// all pairs (tests of the choice: Operator::autotune):
// Row kernels.  FP32: V0 16/512/2, V1 16/256/4, V2 8/256/4; FP64: V0
// 16/512/1, V1 16/256/2, V2 8/256/3.  V3: the small CTAs of small grids (64
// threads, 8 points, 4 up to 128 points per row), which put a grid of 64 to
// 512 rows on all the SMs (FP64 Ns = 128, the forward pass: 5.4 us with
// 16-point threads in 512-thread CTAs, 1.7 us); from 1024 points on 8/512/2,
// two rows of 2048 FP64 points per CTA in runs twice as long (periodic 4096
// apply 268 us with V2, 263).  Sides of 3 2^k: V2 24/128/4 (FP64 2), the
// others 24/256/2 (1).
template <typename T>
__host__ __device__ constexpr int row_rpt(int LR, int v) {
    if (LR % 3 == 0) return 24;
    int want = v == 3 ? (LR <= 128 ? 4 : 8) : (v == 2 ? 8 : 16);
    if (want < LR / 1024) want = LR / 1024;  // at most 1024 threads per transform
    return LR < want ? LR : want;
}
template <typename T>
__host__ __device__ constexpr int row_target_threads(int LR, int v) {
    if (LR % 3 == 0) return v == 2 ? 128 : 256;
    return v == 0 ? 512 : (v == 3 ? (LR >= 1024 ? 512 : 64) : 256);
}
template <typename T>
__host__ __device__ constexpr int row_minb_req(int LR, int v) {
    if (LR % 3 == 0) return (sizeof(T) == 4 ? 2 : 1) * (v == 2 ? 2 : 1);
    const bool wide = v == 3 && LR >= 1024;
    return sizeof(T) == 4 ? (v == 0 || wide ? 2 : (v == 3 ? 1 : 4))
                          : (v == 1 || wide ? 2 : (v == 2 ? 3 : 1));
}
template <typename T>
__host__ __device__ constexpr int row_rb_v(int LR, int v) {
    const int tt = LR / row_rpt<T>(LR, v);
    int rb = row_target_threads<T>(LR, v) / tt;
    if (rb < 1) rb = 1;
    if (rb > 16) rb = 16;
    const int per_row = sm_len(LR + 1) * (int)sizeof(cplx<T>);
    const int mb = row_minb_req<T>(LR, v);
    while (rb > 1 && rb * per_row * mb > kSmemPerSM) rb >>= 1;
    return rb;
}
template <typename T>
__host__ __device__ constexpr int row_threads(int LR, int v) {
    return row_rb_v<T>(LR, v) * (LR / row_rpt<T>(LR, v));
}
template <typename T>
__host__ __device__ constexpr int row_smem_v(int LR, int v) {
    return row_rb_v<T>(LR, v) * sm_len(LR + 1) * (int)sizeof(cplx<T>);
}
template <typename T>
__host__ __device__ constexpr int row_minb(int LR, int v) {
    int mb = row_minb_req<T>(LR, v);
    while (mb > 1 && mb * row_smem_v<T>(LR, v) > kSmemPerSM) --mb;
    while (mb > 1 && mb * row_threads<T>(LR, v) > 1024) --mb;  // 64 registers or more
    return mb;
}

// Column kernel.  FP32: V0 16/<=512/1, V1 16/<=256/3, V2 32/<=256/2 (512/1
// from 8192 points on); FP64: V0 16/<=512/1, V1 16/<=256/2, V2 32/<=256/1; V3
// small CTAs (4 points and 64 threads up to 256 points, then 8 and 128).
// 32 points per thread (one round trip less) against V0: 4096 points FP32
// 43.3 -> 37.9 us, 8192 points 208 -> 186, FP64 8192 points 385 -> 340.
template <typename T>
__host__ __device__ constexpr int col_rpt(int LC, int v) {
    if (LC % 3 == 0) return 24;
    int want = v == 3 ? (LC <= 256 ? 4 : 8) : (v == 2 && LC >= 1024 ? 32 : 16);
    if (want < LC / 1024) want = LC / 1024;  // at most 1024 threads per transform
    return LC < want ? LC : want;
}
template <typename T>
__host__ __device__ constexpr int col_max_threads(int LC, int v) {
    if (LC % 3 == 0) return v == 2 ? 128 : 256;
    return v == 0 ? 512
           : v == 3 ? (LC <= 256 ? 64 : 128)
           : v == 2 && sizeof(T) == 4 && LC >= 8192 ? 512 : 256;
}
template <typename T>
__host__ __device__ constexpr int col_minb_req(int LC, int v) {
    if (LC % 3 == 0) return (sizeof(T) == 4 ? 2 : 1) * (v == 2 ? 2 : 1);
    return sizeof(T) == 4 ? (v == 1 ? 3 : (v == 2 && LC < 8192 ? 2 : 1)) : (v == 1 ? 2 : 1);
}
template <typename T>
__host__ __device__ constexpr int col_ct_v(int LC, int ncols_minus1, int v) {
    const int tt = LC / col_rpt<T>(LC, v);
    const int mb = col_minb_req<T>(LC, v);
    int ct = 16;
    while (ct > 1 && (ct * tt > col_max_threads<T>(LC, v) ||
                      (ct * sm_len(LC) + ct) * (int)sizeof(cplx<T>) * mb > kSmemPerSM ||
                      ct > ncols_minus1))
        ct >>= 1;
    return ct;
}
template <typename T>
__host__ __device__ constexpr int col_smem(int LC, int ct) {
    return (ct * sm_len(LC) + ct) * (int)sizeof(cplx<T>);
}
template <typename T>
__host__ __device__ constexpr int col_threads(int LC, int ncm1, int v) {
    return col_ct_v<T>(LC, ncm1, v) * (LC / col_rpt<T>(LC, v));
}
template <typename T>
__host__ __device__ constexpr int col_minb(int LC, int ncm1, int v) {
    int mb = col_minb_req<T>(LC, v);
    const int sm = col_smem<T>(LC, col_ct_v<T>(LC, ncm1, v));
    while (mb > 1 && mb * sm > kSmemPerSM) --mb;
    while (mb > 1 && mb * col_threads<T>(LC, ncm1, v) > 1024) --mb;
    return mb;
}
// does a column of length LC fit one CTA at all (variant-independent floor)
template <typename T>
__host__ __device__ constexpr bool col_fits(int LC) {
    return col_smem<T>(LC, 1) <= kSmemPerSM;
}

// ---- software pipeline ----------------------------------------------------------
// Where a staging buffer fits beside the FFT workspace of an unpadded column
// tile, the column kernel is persistent -- a CTA walks tiles blockIdx.x,
// blockIdx.x + gridDim.x, ... -- and the next tile is copied global -> shared
// with cp.async while the current one is being transformed.  The waits are
// the hardware's own (cp.async.wait_all): no software spin.  The zero-padded
// columns process one tile per CTA: the loop and the staging cost them
// registers and resident CTAs.  The row passes do so too: staging them (RB
// raw rows, or the tile chunks of RB rows) took 11.5 / 12.7 us at Ns = 2048
// periodic FP32 against 10.4 / 10.0 us with four CTAs per SM.
__host__ __device__ constexpr int align16(int b) { return (b + 15) & ~15; }

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}
// Column: staging of one tile (its stored rows x CT columns, contiguous).
template <typename T, int LC, int NCM1, bool PAD, int V>
__host__ __device__ constexpr int col_stage_bytes() {
    return (PAD ? LC / 2 : LC) * col_ct_v<T>(LC, NCM1, V) * (int)sizeof(cplx<T>);
}
template <typename T, int LC, int NCM1, bool PAD, int V>
__host__ __device__ constexpr bool col_staged() {
    return !PAD && (align16(col_smem<T>(LC, col_ct_v<T>(LC, NCM1, V))) +
            col_stage_bytes<T, LC, NCM1, PAD, V>()) *
               col_minb<T>(LC, NCM1, V) <= kSmemPerSM;
}
// Unstaged column kernels take a second FFT workspace (ping-pong round
// trips, one barrier each instead of two) where it fits beside the CTAs per
// SM the variant asks for.
template <typename T, int LC, int NCM1, bool PAD, int V>
__host__ __device__ constexpr bool col_pp() {
    return !col_staged<T, LC, NCM1, PAD, V>() &&
           2 * align16(col_smem<T>(LC, col_ct_v<T>(LC, NCM1, V))) * col_minb<T>(LC, NCM1, V) <=
               kSmemPerSM;
}
template <typename T, int LC, int NCM1, bool PAD, int V>
__host__ __device__ constexpr int col_smem_total() {
    return col_staged<T, LC, NCM1, PAD, V>()
               ? align16(col_smem<T>(LC, col_ct_v<T>(LC, NCM1, V))) +
                     col_stage_bytes<T, LC, NCM1, PAD, V>()
           : col_pp<T, LC, NCM1, PAD, V>()
               ? 2 * align16(col_smem<T>(LC, col_ct_v<T>(LC, NCM1, V)))
               : col_smem<T>(LC, col_ct_v<T>(LC, NCM1, V));
}

// A load or store with kBatch moves all of a thread's pairs in one call
// (all<count, TT>(row, t, v): pairs t + m TT, m < count) after a begin() that
// reads its scalars: the steps of the PK iteration (pk_device.cuh).  Such a
// store gets the contact mask of its pairs as well, two bits each, which the
// kernel reads ahead of the spectrum.
template <class F, class = void>
struct is_batch : std::false_type {};
template <class F>
struct is_batch<F, std::enable_if_t<F::kBatch>> : std::true_type {};
__device__ __forceinline__ uint32_t pair_mask(uint32_t mb, int k) { return mb >> (2 * k) & 3u; }

// CTAs per SM of an inverse row pass with store F: with a step of the PK
// iteration an FP32 pass gets 80 registers (FP64 fields: 128) instead of 64,
// where it spilled 28-220 bytes
template <typename T, class F>
__host__ __device__ constexpr int row_minb_f(int LR, int v) {
    int mb = row_minb<T>(LR, v);
    if constexpr (is_batch<F>::value) {
        constexpr int regs = sizeof(typename F::Real) == 8 ? 128 : 80;
        while (mb > 1 && mb * row_threads<T>(LR, v) * regs > 65536) --mb;
    }
    return mb;
}

// ---- row forward ---------------------------------------------------------------
// Load:  cplx<T> operator()(int row, int n) -> z[n] = (x[2n], x[2n+1]);
// Store: void operator()(int row, int k, cplx<T> X), k in [0, LR]; with
//        static constexpr bool kTiled (the tiled half spectrum) the kernel
//        writes the tiles through base / nrows / ct / bs itself;
//        static constexpr bool kFinish: when true, every thread
//        calls finish(double* scratch) once, after a __syncthreads() at the end
// Dynamic shared memory: row_smem_v<T>(LR, V).
//
// One group of RB rows per CTA, the row the fastest thread index: RB threads
// and the ct columns of a tile's row then make one contiguous run, so the
// spectrum goes from the registers straight to its tile (RB ct elements per
// run) and only Z[-k], another thread's, comes through shared memory.  The
// pass is bound by L1 (its throughput 75 % in FP32, the shared-memory data
// pipe 60 %, issue 48 %): reading Z[k] from shared memory as well and storing
// by chunk cost one shared pass in seven.  Per launch in back-to-back applies,
// before / after: FP32 Ns = 2048 22.2 / 20.6 us, 4096 148.6 / 80.5, FP64 2048
// 43.0 / 43.9, 4096 196 / 185.
template <typename T, int LR, bool PAD, int V, class Load, class Store>
__global__ void __launch_bounds__(row_threads<T>(LR, V), row_minb<T>(LR, V))
row_fwd_kernel(Load ld, Store st, int nrows, const cplx<T>* __restrict__ tw_lr,
               const cplx<T>* __restrict__ tw_2lr, const int* gate) {
    pdl_wait();
    if (gate && gate[blockIdx.y * kGateStride]) return;
    constexpr int RPT = row_rpt<T>(LR, V);
    constexpr int TT = LR / RPT;
    constexpr int RB = row_rb_v<T>(LR, V);
    extern __shared__ __align__(16) unsigned char smraw[];
    cplx<T>* sm = reinterpret_cast<cplx<T>*>(smraw);
    const int r = threadIdx.x % RB, t = threadIdx.x / RB;
    const int row = blockIdx.x * RB + r;
    const bool valid = row < nrows;
    cplx<T> v[RPT];
    if constexpr (is_batch<Load>::value) {
#pragma unroll
        for (int m = 0; m < RPT; ++m) v[m] = mk<T>(0, 0);
        ld.begin();
        if (valid) ld.template all<(PAD && RPT > 1 ? RPT / 2 : RPT), TT>(row, t, v);
    } else {
#pragma unroll
        for (int m = 0; m < RPT; ++m) {
            if (PAD && m >= RPT / 2) v[m] = mk<T>(0, 0);
            else v[m] = valid ? ld(row, t + m * TT) : mk<T>(0, 0);
        }
    }
    block_fft<T, LR, RPT, -1, RB, PAD>(v, t, sm, r, tw_lr);
#pragma unroll
    for (int m = 0; m < RPT; ++m) sm[smaddr_run<TT, 1 << 30>(t, m, RB, r)] = v[m];
    if (t == 0) sm[smaddr(LR, RB, r)] = v[0];  // Z[LR] = Z[0]: Z[-0] without a mask
    __syncthreads();
    // split step of the real transform: X[k] = E + w^k O with
    // E = (Z[k] + conj Z[-k])/2, O = (Z[k] - conj Z[-k])/(2i), k in [0, LR)
    auto split = [&](int m) {
        const int k = t + m * TT;
        const cplx<T> zk = v[m], zn = sm[smaddr(LR - k, RB, r)], w = __ldg(&tw_2lr[k]);
        const cplx<T> A = mk<T>(zk.x + zn.x, zk.y - zn.y);
        const cplx<T> B = mk<T>(zk.x - zn.x, zk.y + zn.y);
        const cplx<T> O = mk<T>(B.y * T(0.5), -B.x * T(0.5));
        return cadd(cscale(A, T(0.5)), cmul(w, O));
    };
    const cplx<T> zr = mk<T>(v[0].x - v[0].y, T(0));  // k == LR (of thread t == 0)
    if (valid) {
        if constexpr (Store::kTiled) {
            const int ct = st.ct, lct = __ffs(ct) - 1;  // ct is a power of two
            const size_t ts = (size_t)st.nrows * ct;
            cplx<T>* base = st.base + blockIdx.y * st.bs + (size_t)row * ct;
            if constexpr (TT % 16 == 0) {  // ct <= 16 divides TT: a fixed step
                cplx<T>* dst = base + (size_t)(t >> lct) * ts + (t & (ct - 1));
#pragma unroll
                for (int m = 0; m < RPT; ++m) dst[m * ((size_t)TT * st.nrows)] = split(m);
            } else {
#pragma unroll
                for (int m = 0; m < RPT; ++m) {
                    const int k = t + m * TT;
                    base[(size_t)(k >> lct) * ts + (k & (ct - 1))] = split(m);
                }
            }
            if (t == 0) base[(size_t)(LR >> lct) * ts] = zr;
        } else {
#pragma unroll
            for (int m = 0; m < RPT; ++m) st(row, t + m * TT, split(m));
            if (t == 0) st(row, LR, zr);
        }
    }
    if constexpr (Store::kFinish) {
        __syncthreads();
        st.finish(reinterpret_cast<double*>(smraw));
    }
}

// ---- row inverse ----------------------------------------------------------------
// Load:  the tiled half spectrum (base / nrows / ct / bs)
// Store: void operator()(int row, int n, cplx<T> z) -> (x[2n], x[2n+1]);
//        static constexpr bool kFinish (see row_fwd_kernel)
// Dynamic shared memory: row_smem_v<T>(LR, V).
//
// One group of RB rows per CTA in the thread order of row_fwd_kernel: X[k]
// comes from its tile into the thread's registers, X[-k] from the thread that
// loaded it through shared memory.  Per launch in back-to-back applies, before
// / after: FP32 Ns = 2048 18.9 / 17.2 us, 4096 118 / 77, FP64 2048 41.8 / 40.5,
// 4096 202 / 188.
template <typename T, int LR, bool PAD, int V, class Load, class Store>
__global__ void __launch_bounds__(row_threads<T>(LR, V), (row_minb_f<T, Store>(LR, V)))
row_inv_kernel(Load ld, Store st, int nrows, const cplx<T>* __restrict__ tw_lr,
               const cplx<T>* __restrict__ tw_2lr, const int* gate) {
    pdl_wait();
    if (gate && gate[blockIdx.y * kGateStride]) return;
    constexpr int RPT = row_rpt<T>(LR, V);
    constexpr int TT = LR / RPT;
    constexpr int RB = row_rb_v<T>(LR, V);
    extern __shared__ __align__(16) unsigned char smraw[];
    cplx<T>* sm = reinterpret_cast<cplx<T>*>(smraw);
    const int r = threadIdx.x % RB, t = threadIdx.x / RB;
    const int row = blockIdx.x * RB + r;
    const bool valid = row < nrows;
    constexpr int NV = PAD && RPT > 1 ? RPT / 2 : RPT;  // pairs kept
    constexpr int NM = is_batch<Store>::value ? NV : 1;
    uint16_t mw[NM];
    uint32_t mb = 0;
    if constexpr (is_batch<Store>::value) {
        static_assert(NV <= 16, "two mask bits per pair");
        st.begin();
        const uint8_t* mp = st.mask + blockIdx.y * st.bs + (size_t)row * st.pitch + 2 * t;
#pragma unroll
        for (int k = 0; k < NV; ++k)
            mw[k] = valid ? *reinterpret_cast<const uint16_t*>(mp + 2 * k * TT) : (uint16_t)0;
    }
    cplx<T> v[RPT];
    {
        const int ct = ld.ct, lct = __ffs(ct) - 1;  // ct is a power of two
        const size_t ts = (size_t)ld.nrows * ct;
        const cplx<T>* base = ld.base + blockIdx.y * ld.bs + (size_t)(valid ? row : 0) * ct;
        if constexpr (TT % 16 == 0) {  // ct <= 16 divides TT: a fixed step
            const cplx<T>* src = base + (size_t)(t >> lct) * ts + (t & (ct - 1));
#pragma unroll
            for (int m = 0; m < RPT; ++m) v[m] = src[m * ((size_t)TT * ld.nrows)];
        } else {
#pragma unroll
            for (int m = 0; m < RPT; ++m) {
                const int k = t + m * TT;
                v[m] = base[(size_t)(k >> lct) * ts + (k & (ct - 1))];
            }
        }
        if (t == 0) sm[smaddr(LR, RB, r)] = base[(size_t)(LR >> lct) * ts];
    }
#pragma unroll
    for (int m = 0; m < RPT; ++m) sm[smaddr_run<TT, 1 << 30>(t, m, RB, r)] = v[m];
    if constexpr (is_batch<Store>::value) {
#pragma unroll
        for (int k = 0; k < NV; ++k) mb |= ((mw[k] & 1u) | (mw[k] >> 7 & 2u)) << (2 * k);
    }
    __syncthreads();
    // inverse split step: Z[k] = A + i B w^-k, A = X[k] + conj X[-k], B = X[k] - conj X[-k]
#pragma unroll
    for (int m = 0; m < RPT; ++m) {
        const int k = t + m * TT;
        const cplx<T> xk = v[m], xn = sm[smaddr(LR - k, RB, r)];
        const cplx<T> A = mk<T>(xk.x + xn.x, xk.y - xn.y);
        const cplx<T> B = mk<T>(xk.x - xn.x, xk.y + xn.y);
        const cplx<T> Bw = cmulc(B, __ldg(&tw_2lr[k]));  // B * exp(+2 pi i k / 2LR)
        v[m] = mk<T>(A.x - Bw.y, A.y + Bw.x);             // A + i Bw
    }
    __syncthreads();
    block_fft<T, LR, RPT, +1, RB>(v, t, sm, r, tw_lr);
    if constexpr (is_batch<Store>::value) {
        if (valid) st.template all<NV, TT>(row, t, v, mb);
    } else {
#pragma unroll
        for (int m = 0; m < RPT; ++m) {
            if (PAD && m >= RPT / 2) continue;
            if (valid) st(row, t + m * TT, v[m]);
        }
    }
    if constexpr (Store::kFinish) {
        __syncthreads();
        st.finish(reinterpret_cast<double*>(smraw));
    }
}

// ---- column forward * multiplier * inverse --------------------------------------
// Mult: cplx<T> operator()(cplx<T> X, int kx, int ky).  nrows: rows of the
// layout; ndata: the rows that hold data (fewer only in the zero-padded
// transform of an embedded operator: the rest read as zero and are not
// written).  One unit = one tile of CT columns; instance blockIdx.y owns
// NCM1/CT + 1 contiguous tiles.
// Dynamic shared memory: col_smem_total<T, LC, NCM1, PAD, V>().
template <typename T, int LC, int NCM1, bool PAD, int V, class Mult>
__global__ void __launch_bounds__(col_threads<T>(LC, NCM1, V), col_minb<T>(LC, NCM1, V))
col_kernel(cplx<T>* __restrict__ spec, int nrows, int ndata, Mult mul,
           const cplx<T>* __restrict__ tw_lc, const int* gate) {
    pdl_wait();
    if (gate && gate[blockIdx.y * kGateStride]) return;
    constexpr int RPT = col_rpt<T>(LC, V);
    constexpr int CT = col_ct_v<T>(LC, NCM1, V);
    constexpr int TT = LC / RPT;
    constexpr int NTILES = NCM1 / CT + 1;
    constexpr bool STAGED = col_staged<T, LC, NCM1, PAD, V>();
    constexpr int ROWS = PAD ? LC / 2 : LC;  // stored rows of a tile
    // second workspace (elements from sm) of the ping-pong form, else 0
    constexpr int ALT = col_pp<T, LC, NCM1, PAD, V>()
                            ? align16(col_smem<T>(LC, CT)) / (int)sizeof(cplx<T>) : 0;
    constexpr int P1 = ALT ? ping_pong_next<LC, RPT>(0) : 0;
    extern __shared__ __align__(16) unsigned char smraw[];
    cplx<T>* sm = reinterpret_cast<cplx<T>*>(smraw);
    cplx<T>* stg = reinterpret_cast<cplx<T>*>(smraw + align16(col_smem<T>(LC, CT)));
    const int c = threadIdx.x % CT, t = threadIdx.x / CT;
    cplx<T>* inst = spec + (size_t)blockIdx.y * NTILES * nrows * CT;
    const bool all = ndata >= ROWS;
    auto issue = [&](int tile) {  // the tile's stored rows -> stg (cp.async)
        if constexpr (STAGED) {
            constexpr int NV = ROWS * CT * (int)sizeof(cplx<T>) / 16;
            const char* src = reinterpret_cast<const char*>(inst + (size_t)tile * nrows * CT);
            char* dst = reinterpret_cast<char*>(stg);
            for (int f = threadIdx.x; f < NV; f += blockDim.x) cp_async16(dst + 16 * f, src + 16 * f);
            cp_async_commit();
        }
    };
    // transform, multiply, inverse and store of tile `tile` from registers v
    auto body = [&](int tile, cplx<T> (&v)[RPT]) {
        cplx<T>* base = inst + (size_t)tile * nrows * CT;
        block_fft<T, LC, RPT, -1, CT, PAD, ALT>(v, t, sm, c, tw_lc);
        const int kx = tile * CT + c;
#pragma unroll
        for (int m = 0; m < RPT; ++m) v[m] = mul(v[m], kx, t + m * TT);
        block_fft<T, LC, RPT, +1, CT, false, ALT, P1>(v, t, sm, c, tw_lc);
#pragma unroll
        for (int m = 0; m < RPT; ++m) {
            if (PAD && m >= RPT / 2) continue;
            // (all rows: no compare per row; 32 points per thread spilled)
            if (!PAD || all || t + m * TT < ndata) base[(size_t)(t + m * TT) * CT + c] = v[m];
        }
    };
    if constexpr (STAGED) {
        // persistent loop: the next tile is staged during this one
        int tile = blockIdx.x;
        if (tile < NTILES) issue(tile);
        for (; tile < NTILES; tile += gridDim.x) {
            cplx<T> v[RPT];
            cp_async_wait_all();
            __syncthreads();
#pragma unroll
            for (int m = 0; m < RPT; ++m) {
                if (PAD && m >= RPT / 2) v[m] = mk<T>(0, 0);
                else v[m] = stg[(t + m * TT) * CT + c];
            }
            __syncthreads();
            if (tile + (int)gridDim.x < NTILES) issue(tile + gridDim.x);
            body(tile, v);
            __syncthreads();  // the workspace is rewritten by the next tile
        }
    } else {
        // one tile per CTA (a loop costs registers the unstaged kernel cannot
        // spare)
        const int tile = blockIdx.x;
        const cplx<T>* base = inst + (size_t)tile * nrows * CT;
        cplx<T> v[RPT];
        if (!PAD || all) {
#pragma unroll
            for (int m = 0; m < RPT; ++m)
                v[m] = PAD && m >= RPT / 2 ? mk<T>(0, 0) : base[(size_t)(t + m * TT) * CT + c];
        } else {
#pragma unroll
            for (int m = 0; m < RPT; ++m)
                v[m] = m >= RPT / 2 || t + m * TT >= ndata ? mk<T>(0, 0)
                                                           : base[(size_t)(t + m * TT) * CT + c];
        }
        body(tile, v);
    }
}

// ---- split column (free space, the length-2LH column too long for one CTA) -------
// The zero-padded column transform of length M = 2 LH is evaluated as two
// length-LH halves.  With x[n] = 0 for n >= LH and w = exp(-2 pi i / M):
//   X[2m] = FFT_LH(x)[m],   X[2m+1] = FFT_LH(w^n x)[m],
// and for the kept outputs n < LH (unnormalised inverse, as col_kernel)
//   y[n] = IFFT_LH(K[2m] X[2m])[n] + w^-n IFFT_LH(K[2m+1] X[2m+1])[n].
// PARITY 0 writes its half to `acc` (a second spectrum-shaped buffer with the
// same tiled layout); PARITY 1 adds it and writes the column in place.  Each
// launch reads the untouched input column, so the two launches run back to
// back on one stream.  One column tile per CTA; shared memory col_smem<T>(LH, CT).
// ALL: every row holds data (ndata == LH).  Compares per row spill: FP64 at
// 8192 points takes 895 and 1055 us without them, 910 and 1189 with.
template <typename T, int LH, int NCM1, int V, int PARITY, bool ALL, class Mult>
__global__ void __launch_bounds__(col_threads<T>(LH, NCM1, V), col_minb<T>(LH, NCM1, V))
col_split_kernel(cplx<T>* __restrict__ spec, cplx<T>* __restrict__ acc, int nrows, int ndata,
                 Mult mul,
                 const cplx<T>* __restrict__ tw_lh, const cplx<T>* __restrict__ tw_m,
                 const int* gate) {
    pdl_wait();
    if (gate && gate[blockIdx.y * kGateStride]) return;
    constexpr int RPT = col_rpt<T>(LH, V);
    constexpr int CT = col_ct_v<T>(LH, NCM1, V);
    constexpr int TT = LH / RPT;
    constexpr int NTILES = NCM1 / CT + 1;
    extern __shared__ __align__(16) unsigned char smraw[];
    cplx<T>* sm = reinterpret_cast<cplx<T>*>(smraw);
    const int c = threadIdx.x % CT, t = threadIdx.x / CT;
    const size_t off = (size_t)blockIdx.y * NTILES * nrows * CT + (size_t)blockIdx.x * nrows * CT;
    cplx<T>* base = spec + off;
    cplx<T>* abase = acc + off;
    cplx<T> v[RPT];
#pragma unroll
    for (int m = 0; m < RPT; ++m) {
        const int n = t + m * TT;
        v[m] = ALL || n < ndata ? base[(size_t)n * CT + c] : mk<T>(0, 0);
        if constexpr (PARITY) v[m] = cmul(v[m], __ldg(&tw_m[n]));
    }
    block_fft<T, LH, RPT, -1, CT>(v, t, sm, c, tw_lh);
    const int kx = blockIdx.x * CT + c;
#pragma unroll
    for (int m = 0; m < RPT; ++m) v[m] = mul(v[m], kx, 2 * (t + m * TT) + PARITY);
    block_fft<T, LH, RPT, +1, CT>(v, t, sm, c, tw_lh);
#pragma unroll
    for (int m = 0; m < RPT; ++m) {
        const size_t i = (size_t)(t + m * TT) * CT + c;
        if (!ALL && t + m * TT >= ndata) continue;
        if constexpr (PARITY) {
            base[i] = cadd(cmulc(v[m], __ldg(&tw_m[t + m * TT])), abase[i]);
        } else {
            abase[i] = v[m];
        }
    }
}

}  // namespace asb
