// Register-resident Stockham FFT for one CTA-cooperative transform.
//
// A length-L complex transform is carried by L/RPT threads, each holding RPT
// elements in registers.  Thread t always holds elements t + m*(L/RPT),
// m = 0..RPT-1 (the "strided pattern") before and after the transform, and
// the output is in natural order.  The transform is the Stockham autosort
// formulation (Govindaraju et al., "High performance discrete Fourier
// transforms on graphics processors", SC'08): stage s with radix R and span
// Ns reads x[j + r L/R], twiddles input r by w_{Ns R}^{r (j mod Ns)}, does a
// radix-R DFT and writes y[(j div Ns) Ns R + (j mod Ns) + r Ns].  Each thread
// runs RPT/R butterflies per stage (j = t + q L/RPT), whose inputs are exactly
// its own strided registers, so only the stage outputs go through shared
// memory; the last stage's outputs land back in the strided pattern and stay
// in registers.  Stages are radix 16, or 32 where a thread holds 32 points (the
// remainder last), so a 4096-point transform makes two shared-memory round
// trips, and an 8192-point one two at radix 32 instead of three.
//
// Shared memory is addressed as (i + i/16) * S + off (i/32 at radix 32): the
// padding breaks the power-of-two strides of the stage writes, S > 1 interleaves S
// independent transforms element by element (the column kernels).
#pragma once

#include "common.cuh"

namespace asb {

// cos / sin and cos / tan of 2 pi k / 32, 0 < k < 16, k != 8, as plain
// mathematical constants
template <typename T>
__device__ __forceinline__ void unit32(int k, T& c, T& s) {
    switch (k) {
        case 1: c = T(0.9807852804032304491262); s = T(0.1950903220161282678483); break;
        case 2: c = T(0.9238795325112867561282); s = T(0.3826834323650897717285); break;
        case 3: c = T(0.8314696123025452370788); s = T(0.5555702330196022247428); break;
        case 4: c = T(0.7071067811865475244008); s = T(0.7071067811865475244008); break;
        case 5: c = T(0.5555702330196022247428); s = T(0.8314696123025452370788); break;
        case 6: c = T(0.3826834323650897717285); s = T(0.9238795325112867561282); break;
        case 7: c = T(0.1950903220161282678483); s = T(0.9807852804032304491262); break;
        case 9: c = T(-0.1950903220161282678483); s = T(0.9807852804032304491262); break;
        case 10: c = T(-0.3826834323650897717285); s = T(0.9238795325112867561282); break;
        case 11: c = T(-0.5555702330196022247428); s = T(0.8314696123025452370788); break;
        case 12: c = T(-0.7071067811865475244008); s = T(0.7071067811865475244008); break;
        case 13: c = T(-0.8314696123025452370788); s = T(0.5555702330196022247428); break;
        case 14: c = T(-0.9238795325112867561282); s = T(0.3826834323650897717285); break;
        case 15: c = T(-0.9807852804032304491262); s = T(0.1950903220161282678483); break;
        default: c = T(0); s = T(1); break;
    }
}
template <typename T>
__device__ __forceinline__ void unit32_cos_tan(int k, T& c, T& t) {
    switch (k) {
        case 1: c = T(0.9807852804032304491262); t = T(0.1989123673796580069116); break;
        case 2: c = T(0.9238795325112867561282); t = T(0.4142135623730950488017); break;
        case 3: c = T(0.8314696123025452370788); t = T(0.6681786379192989199978); break;
        case 4: c = T(0.7071067811865475244008); t = T(1.0); break;
        case 5: c = T(0.5555702330196022247428); t = T(1.496605762665489017601); break;
        case 6: c = T(0.3826834323650897717285); t = T(2.414213562373095048802); break;
        case 7: c = T(0.1950903220161282678483); t = T(5.027339492125848104515); break;
        case 9: c = T(-0.1950903220161282678483); t = T(-5.027339492125848104515); break;
        case 10: c = T(-0.3826834323650897717285); t = T(-2.414213562373095048802); break;
        case 11: c = T(-0.5555702330196022247428); t = T(-1.496605762665489017601); break;
        case 12: c = T(-0.7071067811865475244008); t = T(-1.0); break;
        case 13: c = T(-0.8314696123025452370788); t = T(-0.6681786379192989199978); break;
        case 14: c = T(-0.9238795325112867561282); t = T(-0.4142135623730950488017); break;
        case 15: c = T(-0.9807852804032304491262); t = T(-0.1989123673796580069116); break;
        default: c = T(1); t = T(0); break;
    }
}

// the same of 2 pi k / 24, 0 < k < 12, k != 6
template <typename T>
__device__ __forceinline__ void unit24(int k, T& c, T& s) {
    switch (k) {
        case 1: c = T(0.9659258262890682867497); s = T(0.2588190451025207623489); break;
        case 2: c = T(0.8660254037844386467637); s = T(0.5); break;
        case 3: c = T(0.7071067811865475244008); s = T(0.7071067811865475244008); break;
        case 4: c = T(0.5); s = T(0.8660254037844386467637); break;
        case 5: c = T(0.2588190451025207623489); s = T(0.9659258262890682867497); break;
        case 7: c = T(-0.2588190451025207623489); s = T(0.9659258262890682867497); break;
        case 8: c = T(-0.5); s = T(0.8660254037844386467637); break;
        case 9: c = T(-0.7071067811865475244008); s = T(0.7071067811865475244008); break;
        case 10: c = T(-0.8660254037844386467637); s = T(0.5); break;
        case 11: c = T(-0.9659258262890682867497); s = T(0.2588190451025207623489); break;
        default: c = T(0); s = T(1); break;
    }
}
template <typename T>
__device__ __forceinline__ void unit24_cos_tan(int k, T& c, T& t) {
    switch (k) {
        case 1: c = T(0.9659258262890682867497); t = T(0.2679491924311227064726); break;
        case 2: c = T(0.8660254037844386467637); t = T(0.5773502691896257645091); break;
        case 3: c = T(0.7071067811865475244008); t = T(1.0); break;
        case 4: c = T(0.5); t = T(1.732050807568877293527); break;
        case 5: c = T(0.2588190451025207623489); t = T(3.732050807568877293527); break;
        case 7: c = T(-0.2588190451025207623489); t = T(-3.732050807568877293527); break;
        case 8: c = T(-0.5); t = T(-1.732050807568877293527); break;
        case 9: c = T(-0.7071067811865475244008); t = T(-1.0); break;
        case 10: c = T(-0.8660254037844386467637); t = T(-0.5773502691896257645091); break;
        case 11: c = T(-0.9659258262890682867497); t = T(-0.2679491924311227064726); break;
        default: c = T(1); t = T(0); break;
    }
}
// the circle that radix R divides: 32 points, or 24 where 3 divides R
__host__ __device__ constexpr int unit_points(int R) { return R % 3 == 0 ? 24 : 32; }

// a * exp(DIR * 2 pi i k / R) for a compile-time R that divides 32 or 24.
template <int R, int DIR, typename T>
__device__ __forceinline__ cplx<T> rot_const(cplx<T> a, int k) {
    constexpr int U = unit_points(R);
    const int ku = k * (U / R);
    if (ku == 0) return a;
    if (ku == U / 4) return mul_i<DIR>(a);
    T c, s;
    if constexpr (U == 24) unit24<T>(ku, c, s);
    else unit32<T>(ku, c, s);
    const T sn = DIR < 0 ? -s : s;
    return mk<T>(a.x * c - a.y * sn, a.x * sn + a.y * c);
}

// The radix-2 butterfly with the odd input rotated by exp(DIR 2 pi i k / R):
// lo = e + w o, hi = e - w o.  A general rotation is factored as
// w o = c (o.x - t o.y, o.y + t o.x), t = tan of the angle (cos c != 0), and
// the factor c is folded into the two outputs' fused multiply-adds: six
// instructions instead of a four-instruction rotation and four additions.
template <int R, int DIR, typename T>
__device__ __forceinline__ void bfly_rot(cplx<T> e, cplx<T> o, int k, cplx<T>& lo, cplx<T>& hi) {
    constexpr int U = unit_points(R);
    const int ku = k * (U / R);
    if (ku == 0) {
        lo = cadd(e, o);
        hi = csub(e, o);
    } else if (ku == U / 4) {
        const cplx<T> w = mul_i<DIR>(o);
        lo = cadd(e, w);
        hi = csub(e, w);
    } else {
        T c, t;
        if constexpr (U == 24) unit24_cos_tan<T>(ku, c, t);
        else unit32_cos_tan<T>(ku, c, t);
        if (DIR < 0) t = -t;
        const T ux = fma(-t, o.y, o.x), uy = fma(t, o.x, o.y);
        lo = mk<T>(fma(c, ux, e.x), fma(c, uy, e.y));
        hi = mk<T>(fma(-c, ux, e.x), fma(-c, uy, e.y));
    }
}

// In-register DFT of R points (natural order in and out), radix-2 DIT split.
template <int R, int DIR, typename T>
__device__ __forceinline__ void dft(cplx<T>* a) {
    if constexpr (R == 1) {
        return;
    } else if constexpr (R == 2) {
        const cplx<T> t = a[0];
        a[0] = cadd(t, a[1]);
        a[1] = csub(t, a[1]);
    } else if constexpr (R == 3) {
        // X0 = a0 + s, X1/2 = a0 - s/2 +- DIR i (sqrt 3 / 2) d, s/d = a1 +- a2
        const T h = T(0.8660254037844386467637);
        const cplx<T> sm = cadd(a[1], a[2]), d = csub(a[1], a[2]);
        const cplx<T> m = mk<T>(fma(T(-0.5), sm.x, a[0].x), fma(T(-0.5), sm.y, a[0].y));
        const cplx<T> r = mul_i<DIR>(d);
        a[0] = cadd(a[0], sm);
        a[1] = mk<T>(fma(h, r.x, m.x), fma(h, r.y, m.y));
        a[2] = mk<T>(fma(-h, r.x, m.x), fma(-h, r.y, m.y));
    } else if constexpr (R == 4) {
        const cplx<T> s02 = cadd(a[0], a[2]), d02 = csub(a[0], a[2]);
        const cplx<T> s13 = cadd(a[1], a[3]);
        const cplx<T> d13 = mul_i<DIR>(csub(a[1], a[3]));
        a[0] = cadd(s02, s13);
        a[2] = csub(s02, s13);
        a[1] = cadd(d02, d13);
        a[3] = csub(d02, d13);
    } else {
        cplx<T> e[R / 2], o[R / 2];
#pragma unroll
        for (int i = 0; i < R / 2; ++i) { e[i] = a[2 * i]; o[i] = a[2 * i + 1]; }
        dft<R / 2, DIR, T>(e);
        dft<R / 2, DIR, T>(o);
#pragma unroll
        for (int k = 0; k < R / 2; ++k) bfly_rot<R, DIR, T>(e[k], o[k], k, a[k], a[k + R / 2]);
    }
}

// The DFT of R points whose upper half a[R/2 .. R-1] is zero (the first
// stage of a zero-padded transform): with w = exp(DIR 2 pi i / R),
//   X[2k] = DFT_{R/2}(a)[k],   X[2k+1] = DFT_{R/2}(a[n] w^n)[k],  n < R/2,
// two half-length DFTs instead of the full one on zeros (x + 0 is not folded
// by the compiler: -0 + 0 = +0).
template <int R, int DIR, typename T>
__device__ __forceinline__ void dft_upper_zero(cplx<T>* a) {
    cplx<T> b[R / 2], c[R / 2];
#pragma unroll
    for (int n = 0; n < R / 2; ++n) {
        b[n] = a[n];
        c[n] = rot_const<R, DIR, T>(a[n], n);
    }
    dft<R / 2, DIR, T>(b);
    dft<R / 2, DIR, T>(c);
#pragma unroll
    for (int k = 0; k < R / 2; ++k) {
        a[2 * k] = b[k];
        a[2 * k + 1] = c[k];
    }
}

__host__ __device__ constexpr int ilog2c(int v) { return v <= 1 ? 0 : 1 + ilog2c(v >> 1); }

// Radix of the stage that has `rem` left to transform, with at most RMAX
// points per thread.  RMAX = 3 2^k (transforms of 3 2^n points): the first
// stage takes the factor 3, the later ones powers of two that divide RMAX.
__host__ __device__ constexpr int next_radix(int rem, int RMAX) {
    const int cap = RMAX % 3 == 0 && rem % 3 != 0 ? RMAX / 3 : RMAX;
    return rem >= cap ? cap : rem;
}
// Radix of stage `s` for a length-L transform with at most RMAX per stage.
__host__ __device__ constexpr int stage_radix(int L, int RMAX, int s) {
    int rem = L;
    for (int i = 0; i < s; ++i) rem /= next_radix(rem, RMAX);
    return next_radix(rem, RMAX);
}
__host__ __device__ constexpr int num_stages(int L, int RMAX) {
    int n = 0, rem = L;
    while (rem > 1) { rem /= next_radix(rem, RMAX); ++n; }
    return n;
}

template <int PS = 4>
__device__ __forceinline__ int smaddr(int i, int S, int off) { return (i + (i >> PS)) * S + off; }

// smaddr(i0 + m * STEP) as a per-thread base plus a compile-time offset where
// the padding term splits.  For STEP a multiple of 16, (i0 + m STEP) >> 4 =
// (i0 >> 4) + m STEP / 16.  RUN is the length (a power of two) of the
// RUN-aligned group that every i0 + m STEP stays in; for RUN <= 16 that group
// lies inside one 16-element block, so the padding term does not change
// with m.
// PS: one element of padding per 2^PS.
template <int STEP, int RUN, int PS = 4>
__device__ __forceinline__ int smaddr_run(int i0, int m, int S, int off) {
    constexpr int PAD1 = 1 << PS;
    if constexpr (STEP % PAD1 == 0) return smaddr<PS>(i0, S, off) + m * (STEP + STEP / PAD1) * S;
    else if constexpr (RUN <= PAD1 && (RUN & (RUN - 1)) == 0) return smaddr<PS>(i0, S, off) + m * STEP * S;
    else return smaddr<PS>(i0 + m * STEP, S, off);
}

// a * w (forward) or a * conj(w) (inverse), w from the exp(-2 pi i k/L) table
template <int DIR, typename V>
__device__ __forceinline__ V tw_apply(V a, V w) {
    return DIR < 0 ? cmul(a, w) : cmulc(a, w);
}

// Shared-memory elements needed by one transform of length L (padded).
__host__ __device__ constexpr int sm_len(int L) { return L + L / 16 + 1; }

template <typename T, int L, int RPT, int DIR, int S, int STAGE, int SPAN, bool HZ, int ALT,
          int P0>
__device__ __forceinline__ void fft_stages(cplx<T> (&v)[RPT], int t, cplx<T>* sm, int off,
                                           const cplx<T>* __restrict__ tw) {
    constexpr int RMAX = RPT < 32 ? RPT : 32;
    // one element of padding per radix of the first stage's writes
    constexpr int PS = RPT < 32 ? 4 : 5;
    constexpr int NST = num_stages(L, RMAX);
    if constexpr (STAGE < NST) {
        constexpr int R = stage_radix(L, RMAX, STAGE);
        constexpr int TT = L / RPT;   // threads per transform
        constexpr int Q = RPT / R;    // butterflies per thread
        constexpr bool LAST = (STAGE == NST - 1);
        static_assert(RPT % R == 0, "radix must divide RPT");
        // this round trip's workspace: with ALT > 0, round trips alternate
        // between sm and sm + ALT, starting at parity P0
        cplx<T>* ws = (ALT > 0 && ((STAGE + P0) & 1)) ? sm + ALT : sm;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int j = t + q * TT;
            cplx<T> a[R];
#pragma unroll
            for (int r = 0; r < R; ++r) a[r] = v[q + r * Q];
            if constexpr (SPAN > 1) {
                // w^r for r = 1..R-1 from the loaded powers w, w^2, w^4, .. w^(R/2)
                // (products at most three deep), applied as each is formed.
                // w^(2^e) = exp(-2 pi i jm / (SPAN R / 2^e)) is entry jm of the
                // length-(SPAN R / 2^e) table, so consecutive threads (jm)
                // read consecutive entries instead of a stride of L/(SPAN R).
                // On the inputs, not folded into the butterflies (lo = e + w o,
                // hi = 2 e - lo): that saves 2 instructions in 15 per point,
                // but hi carries lo's rounding as well and a point passes
                // log2 R rounded twiddles.  Against 64 bits an FP32 apply of a
                // positive field was 18-35 % further off than pocketfft's FP32
                // so, 2-16 % is; solves in FP32 stagnated a fifth higher.
                // Free-space apply, folded / on the inputs: FP32 2048 71.9 /
                // 72.5 us, 4096 326 / 340, FP64 4096 724 / 708.
                const int jm = j % SPAN;
                const cplx<T>* __restrict__ tb = tw - L;  // tables at offset = length
                auto power = [&](int e) { return __ldg(&tb[SPAN * R / e + jm]); };
                // w .. w^(LOW-1) stay in registers: three at radix 16 (seven
                // spill in the FP64 column kernels), seven at 32 (4 % of the
                // FP32 apply at 4096, 1.5 % of the FP64 one)
                constexpr int LOW = R > 16 ? 8 : (R < 4 ? R : 4);
                cplx<T> w[LOW], wa = mk<T>(T(0), T(0)), wb = wa;
#pragma unroll
                for (int r = 1; r < LOW; ++r) {
                    w[r] = (r & (r - 1)) == 0 ? power(r) : cmul(w[r > 4 ? 4 : 2], w[r > 4 ? r - 4 : 1]);
                    a[r] = tw_apply<DIR>(a[r], w[r]);
                }
#pragma unroll
                for (int h = LOW; h < R; h += LOW) {
                    cplx<T> wh;
                    if (h == LOW) wh = wa = power(h);
                    else if (h == 2 * LOW) wh = wb = power(h);
                    else wh = cmul(wb, wa);
                    a[h] = tw_apply<DIR>(a[h], wh);
#pragma unroll
                    for (int r = 1; r < LOW; ++r) a[h + r] = tw_apply<DIR>(a[h + r], cmul(wh, w[r]));
                }
            }
            // the zero upper half of the input (HZ) is the upper half of
            // every first-stage butterfly: a[r] = v[q + r Q] with v[m] = 0
            // for m >= RPT / 2 exactly when r >= R / 2
            if constexpr (HZ && STAGE == 0 && R >= 2)
                dft_upper_zero<R, DIR, T>(a);
            else
                dft<R, DIR, T>(a);
            if constexpr (LAST) {
#pragma unroll
                for (int r = 0; r < R; ++r) v[q + r * Q] = a[r];
            } else {
                const int base = (j / SPAN) * SPAN * R + (j % SPAN);
#pragma unroll
                for (int r = 0; r < R; ++r) ws[smaddr_run<SPAN, SPAN * R, PS>(base, r, S, off)] = a[r];
            }
        }
        if constexpr (!LAST) {
            __syncthreads();
#pragma unroll
            for (int m = 0; m < RPT; ++m) v[m] = ws[smaddr_run<TT, 1 << 30, PS>(t, m, S, off)];
            // one workspace: nobody writes it again before everyone has read
            // it.  Two (ALT > 0): the next round trip writes the other one,
            // and the one after that follows the next round trip's barrier,
            // which every thread reaches only after this read.
            if constexpr (ALT == 0) __syncthreads();
            fft_stages<T, L, RPT, DIR, S, STAGE + 1, SPAN * R, HZ, ALT, P0>(v, t, sm, off, tw);
        }
    }
}

// Length-L transform (L = 2^n, or 3 2^n with RPT = 24) of the strided
// register pattern; DIR = -1 forward
// (exp(-2 pi i jk/L)), +1 inverse, both unnormalised.  tw points at the
// length-L table exp(-2 pi i k / L), k < L, inside one array that holds the
// table of every length M = L / 2^j at offset M (so tw - L is the
// array base and the stages read the shorter tables).  Every thread of the CTA must
// call this (it contains __syncthreads), including threads whose transform
// is a dummy.  HZ: the upper half of the input is zero (v[m] = 0 for
// m >= RPT / 2, a zero-padded transform); its first stage skips the zeros.
// ALT > 0: a second workspace of the same shape at sm + ALT (elements); the
// shared-memory round trips alternate between the two, which saves the
// barrier after each read.  The first round trip uses parity P0 (0: sm,
// 1: sm + ALT); a caller that runs two transforms back to back without a
// barrier between them starts the second at ping_pong_next<L, RPT>(P0), the
// workspace the first one did not read last.
template <typename T, int L, int RPT, int DIR, int S, bool HZ = false, int ALT = 0, int P0 = 0>
__device__ __forceinline__ void block_fft(cplx<T> (&v)[RPT], int t, cplx<T>* sm, int off,
                                          const cplx<T>* __restrict__ tw) {
    static_assert(L % RPT == 0, "L must be a multiple of RPT");
    fft_stages<T, L, RPT, DIR, S, 0, 1, HZ, ALT, P0>(v, t, sm, off, tw);
}

// parity of the first round trip after a ping-pong transform that started at
// P0: the workspace its last round trip did not read
template <int L, int RPT>
__host__ __device__ constexpr int ping_pong_next(int p0) {
    return (p0 + num_stages(L, RPT < 32 ? RPT : 32) - 1) & 1;
}

}  // namespace asb
