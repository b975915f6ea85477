// ld_fxpass.cuh — Stockham stages of compile-time length and radix order, the
// first stage fed from, and the last drained to, wherever the pass keeps its
// data: global memory, staged bulk copies, a spectral product, a converted
// store.  A pass of three stages then moves each value through shared memory
// twice instead of five times (fill, three in-place stages, drain).  The
// length, the radix and span of every stage and the thread count are
// constants, so a butterfly's addresses are one base plus immediate offsets
// and its divisions are by constants; the twiddles w^r of butterfly k come from
// a per-stage table of pairs (w^2q, w^(2q+1)) laid out [q][k], read as 16-byte
// loads that a warp's threads (consecutive k) make to consecutive addresses
// (fx_stage_table in ld_frame_fx.cu).
//
// A stage of radix R over span NS takes butterfly b = j * C + c (j < N / R,
// sequence c of C interleaved ones): its inputs are the elements
// e = b + r * (N / R) * C of the sequences laid out [index][sequence], its
// outputs ((j - k) * R + k + r * NS) * C + c, k = j mod NS.  The last stage
// has NS = N / R, so its outputs are again b + r * (N / R) * C: a thread's
// values of the last stage are N / R rows apart, consecutive threads hold
// consecutive (row, sequence) pairs.
#pragma once

#include <atomic>

#include "ld_async.cuh"
#include "ld_fft.cuh"
#include "ld_fxorder.h"
#include "ld_internal.h"
#include "ld_launch.cuh"

namespace ld {

template <int R>
struct FxPad {  // a stage table holds an even number of twiddles per span offset
    static constexpr int value = (R + 1) & ~1;
};

// ---- small DFTs of the composite radices --------------------------------------
// cos and sin of 2 pi m / R to double precision at compile time: the argument
// folded to an eighth of a turn, then the Taylor series.
struct UnitRoot {
    double c, s;
};
__host__ __device__ constexpr UnitRoot unit_root(int m, int R) {
    m %= R;
    int n8 = 8 * m;  // the angle in eighths of a turn, times R
    const int oct = n8 / R;
    n8 -= oct * R;
    const double frac = static_cast<double>(n8) / R;  // in [0, 1): eighths of a turn past `oct`
    const bool odd = (oct & 1) != 0;
    const double x = (odd ? 1.0 - frac : frac) * 0.78539816339744830962;
    double c = 0.0, s = 0.0, t = 1.0;
    for (int i = 0; i < 24; ++i) {  // t = x^i / i!
        if ((i & 1) == 0) c += (i & 2) ? -t : t;
        else s += (i & 2) ? -t : t;
        t *= x / (i + 1);
    }
    // (c, s) is the root of x in [0, pi / 4]; odd octants mirror it about pi / 4
    const double a = odd ? s : c, b = odd ? c : s;
    switch (oct / 2) {
        case 0: return {a, b};
        case 1: return {-b, a};
        case 2: return {-a, -b};
        default: return {b, -a};
    }
}

// x * exp(-+ 2 pi i E / R) (forward / INV), E a compile-time exponent.
template <int R, int E, bool INV>
__device__ __forceinline__ float2 rotate(float2 x) {
    constexpr int e = ((E % R) + R) % R;
    if constexpr (e == 0) {
        return x;
    } else if constexpr (4 * e == R) {
        return rot90<INV>(x);
    } else if constexpr (2 * e == R) {
        return make_float2(-x.x, -x.y);
    } else if constexpr (4 * e == 3 * R) {
        return rot90<!INV>(x);
    } else {
        constexpr UnitRoot u = unit_root(e, R);
        constexpr float c = static_cast<float>(u.c), s = static_cast<float>(INV ? u.s : -u.s);
        return make_float2(x.x * c - x.y * s, x.x * s + x.y * c);
    }
}

template <int R, bool INV>
__device__ __forceinline__ void fdft(float2* v);

template <int A, int B, bool INV, int R2, int... K1>
__device__ __forceinline__ void fdft_col(float2* v, std::integer_sequence<int, K1...>) {
    float2 t[A];
#pragma unroll
    for (int r1 = 0; r1 < A; ++r1) t[r1] = v[B * r1 + R2];
    fdft<A, INV>(t);
    ((v[B * K1 + R2] = rotate<A * B, R2 * K1, INV>(t[K1])), ...);
}
template <int A, int B, bool INV, int... R2>
__device__ __forceinline__ void fdft_cols(float2* v, std::integer_sequence<int, R2...>) {
    (fdft_col<A, B, INV, R2>(v, std::make_integer_sequence<int, A>{}), ...);
}

// Radix A * B in registers (r = B r1 + r2, k = k1 + A k2): DFT-A over r1, the
// inner twiddles, DFT-B over r2.
template <int A, int B, bool INV>
__device__ __forceinline__ void fdft_composite(float2* v) {
    fdft_cols<A, B, INV>(v, std::make_integer_sequence<int, B>{});
    float2 o[A * B];
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
        float2 t[B];
#pragma unroll
        for (int r2 = 0; r2 < B; ++r2) t[r2] = v[B * k1 + r2];
        fdft<B, INV>(t);
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) o[k1 + A * k2] = t[k2];
    }
#pragma unroll
    for (int r = 0; r < A * B; ++r) v[r] = o[r];
}

template <int R, bool INV>
__device__ __forceinline__ void fdft(float2* v) {
    if constexpr (R == 2) dft2<INV>(v);
    else if constexpr (R == 3) dft3<INV>(v);
    else if constexpr (R == 4) dft4<INV>(v);
    else if constexpr (R == 5) dft5<INV>(v);
    else if constexpr (R == 8) dft8<INV>(v);
    else if constexpr (R == 9) fdft_composite<3, 3, INV>(v);
    else if constexpr (R == 10) fdft_composite<5, 2, INV>(v);
    else if constexpr (R == 12) fdft_composite<3, 4, INV>(v);
    else if constexpr (R == 15) fdft_composite<5, 3, INV>(v);
    else if constexpr (R == 16) fdft_composite<4, 4, INV>(v);
    else if constexpr (R == 20) fdft_composite<5, 4, INV>(v);
    else if constexpr (R == 24) fdft_composite<3, 8, INV>(v);
    else fdft_composite<5, 5, INV>(v);
}

// ---- stages ---------------------------------------------------------------------
// The twiddles of one butterfly of span offset k (NS = 1: none).
template <bool INV, int R, int NS>
__device__ __forceinline__ void fp_twiddle(float2* v, int k, const float2* __restrict__ stw) {
    if constexpr (NS > 1) {
        const float4* t = reinterpret_cast<const float4*>(stw) + k;
#pragma unroll
        for (int q = 0; q < FxPad<R>::value / 2; ++q) {
            const float4 w = __ldg(t + q * NS);
            if (q > 0) v[2 * q] = INV ? cmulc(v[2 * q], make_float2(w.x, w.y)) : cmul(v[2 * q], make_float2(w.x, w.y));
            if (2 * q + 1 < R) {
                const float2 w1 = make_float2(w.z, w.w);
                v[2 * q + 1] = INV ? cmulc(v[2 * q + 1], w1) : cmul(v[2 * q + 1], w1);
            }
        }
    }
}

// How a stage takes a butterfly of span offset k.  FastStage: the radices of
// ld_fxplans.h.
struct FastStage {
    template <bool INV, int R, int NS>
    static __device__ __forceinline__ void run(float2* v, int k, const float2* __restrict__ stw) {
        fp_twiddle<INV, R, NS>(v, k, stw);
        fdft<R, INV>(v);
    }
};
// A pass of ld_fxorder.h: the stage of radix A over span NS and (B > 1) the
// stage of radix B over span NS * A after it, with the arithmetic of
// ld_fft.cuh.  The B butterflies j, j + N / (A B), .. of the first (inputs r
// = B r1 + r2) feed the A butterflies of span offsets k1 NS + k of the second.
template <int A, int B>
struct OrderStage {
    template <bool INV, int R, int NS>
    static __device__ __forceinline__ void run(float2* v, int k, const float2* __restrict__ stw) {
        static_assert(R == A * B);
        if constexpr (B == 1) {
            fp_twiddle<INV, A, NS>(v, k, stw);
            dft<A, INV>(v);
        } else {
#pragma unroll
            for (int r2 = 0; r2 < B; ++r2) {
                float2 t[A];
#pragma unroll
                for (int r1 = 0; r1 < A; ++r1) t[r1] = v[B * r1 + r2];
                fp_twiddle<INV, A, NS>(t, k, stw);
                dft<A, INV>(t);
#pragma unroll
                for (int k1 = 0; k1 < A; ++k1) v[B * k1 + r2] = t[k1];
            }
            const float2* second = stw + FxOrder::stage(NS, A);
            float2 o[R];
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1) {
                float2 t[B];
#pragma unroll
                for (int r2 = 0; r2 < B; ++r2) t[r2] = v[B * k1 + r2];
                fp_twiddle<INV, B, NS * A>(t, k1 * NS + k, second);
                dft<B, INV>(t);
#pragma unroll
                for (int k2 = 0; k2 < B; ++k2) o[k1 + A * k2] = t[k2];
            }
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = o[r];
        }
    }
};

// One stage: ld(e) gives element e, st(e, value) takes it; SYNC: a CTA barrier
// between the last load and the first store (the two share a buffer).
template <int N, int C, int T, bool INV, int R, int NS, bool SYNC, class Stage = FastStage, class Ld, class St>
__device__ __forceinline__ void fp_stage(const float2* __restrict__ stw, Ld ld, St st) {
    constexpr int NB = N / R * C;
    constexpr int IT = (NB + T - 1) / T;
    const int tid = static_cast<int>(threadIdx.x);
    float2 v[IT][R];
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int b = tid + it * T;
        if ((it + 1) * T <= NB || b < NB) {
#pragma unroll
            for (int r = 0; r < R; ++r) v[it][r] = ld(b + r * NB);
        }
    }
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int b = tid + it * T;
        if ((it + 1) * T <= NB || b < NB) Stage::template run<INV, R, NS>(v[it], (b / C) % NS, stw);
    }
    if constexpr (SYNC) __syncthreads();
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int b = tid + it * T;
        if ((it + 1) * T <= NB || b < NB) {
            const int j = b / C;
            const int k = j % NS;
            const int base = ((j - k) * R + k) * C + (b - j * C);
#pragma unroll
            for (int r = 0; r < R; ++r) st(base + r * NS * C, v[it][r]);
        }
    }
}

// The last stage, kept in the thread's registers: v[it][r] is element
// tid + it * T + r * NB where that butterfly exists.
template <int N, int C, int T, bool INV, int R, class Stage = FastStage>
struct LastStage {
    static constexpr int NB = N / R * C;
    static constexpr int IT = (NB + T - 1) / T;
    float2 v[IT][R];
    static __device__ __forceinline__ bool has(int it) {
        return (it + 1) * T <= NB || static_cast<int>(threadIdx.x) + it * T < NB;
    }
    template <class Ld>
    __device__ __forceinline__ void run(const float2* __restrict__ stw, Ld ld) {
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int b = static_cast<int>(threadIdx.x) + it * T;
            if (has(it)) {
#pragma unroll
                for (int r = 0; r < R; ++r) v[it][r] = ld(b + r * NB);
            }
        }
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int b = static_cast<int>(threadIdx.x) + it * T;
            if (has(it)) Stage::template run<INV, R, N / R>(v[it], b / C, stw);
        }
    }
    // f(e, value) for every element the thread holds
    template <class F>
    __device__ __forceinline__ void each(F f) const {
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int b = static_cast<int>(threadIdx.x) + it * T;
            if (has(it)) {
#pragma unroll
                for (int r = 0; r < R; ++r) f(b + r * NB, v[it][r]);
            }
        }
    }
};

// A three-stage transform length; ord: the FP16 form's order.
template <int R1_, int R2_, int R3_>
struct Fx3 {
    static constexpr int R1 = R1_, R2 = R2_, R3 = R3_;
    static constexpr int n = R1 * R2 * R3;
    // stage tables follow one another: the second stage's, then the third's,
    // then the order's (fx_stage_table in ld_frame_fx.cu)
    static constexpr int tab2 = 0, tab3 = R1 * FxPad<R2>::value;
    static constexpr int tab_ord = tab3 + R1 * R2 * FxPad<R3>::value;
    static constexpr FxOrder ord = fx_col_order(R1, R2, R3);
    static constexpr bool table_twiddles = fx_table_twiddles(false, n);
};

// Where the order's twiddles lie: by products, then (lengths that have them)
// from the table, which the spectral chain takes.
template <class P, bool SPECTRAL>
__device__ __forceinline__ const float2* ord_table(const float2* stw) {
    return stw + P::tab_ord + (SPECTRAL && P::table_twiddles ? P::ord.table() : 0);
}

// Pass I of P's order.
template <class P, int I>
using OrdStage = OrderStage<P::ord.a[I], P::ord.b[I]>;
template <class P, int C, int T, bool INV, int I, bool SYNC, class Ld, class St>
__device__ __forceinline__ void ord_pass(const float2* __restrict__ tw, Ld ld, St st) {
    fp_stage<P::n, C, T, INV, P::ord.radix(I), P::ord.span(I), SYNC, OrdStage<P, I>>(tw + P::ord.table(I), ld, st);
}
// The passes from I to the one before the last, in place in s, a barrier after each.
template <class P, int C, int T, bool INV, int I = 1>
__device__ __forceinline__ void ord_middle(const float2* __restrict__ tw, float2* s) {
    if constexpr (I < P::ord.count - 1) {
        ord_pass<P, C, T, INV, I, true>(tw, [&](int e) { return s[e]; }, [&](int e, float2 v) { s[e] = v; });
        __syncthreads();
        ord_middle<P, C, T, INV, I + 1>(tw, s);
    }
}
// The last pass, in registers.
template <class P, int C, int T, bool INV>
using OrdLast = LastStage<P::n, C, T, INV, P::ord.radix(P::ord.count - 1), OrdStage<P, P::ord.count - 1>>;

// Largest m over the CTA of T threads (every thread gets it); `part`: a shared
// array of at least T / 32 floats, nobody's until the next barrier.
template <int T>
__device__ __forceinline__ float cta_max(float m, float* part) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < T / 32; ++w) m = fmaxf(m, part[w]);
    return m;
}

// The Mono (three drivers, one kernel) and luma-lock (four kernels) chains are
// compiled for lengths up to this one, every HD and most UHD grids: there their
// column passes take 193 us (Mono) and 143 us, against 313 and 223 on the
// runtime-planned transforms.  Longer ones would gain too; they are left out to
// keep the library (105 MB, built in two minutes) from growing for the largest
// frames of these two chains.
constexpr int kFxOtherMax = 3200;

// Largest dynamic shared memory of a kernel without static shared memory.
constexpr size_t kSmemOptIn = 227 * 1024;

// A kernel's per-device launch state, set up at its first launch on a device:
// the dynamic shared-memory opt-in and the CTAs resident at once.
struct KernelState {
    std::atomic<int> resident[16] = {};
    template <class K>
    int get(K kernel, int threads, size_t smem) {
        int dev = 0;
        cudaGetDevice(&dev);
        const int known = dev < 16 ? resident[dev].load(std::memory_order_relaxed) : 0;
        if (known > 0) return known;
        int sms = 148, per = 1;
        cudaFuncAttributes fa{};
        cudaFuncGetAttributes(&fa, kernel);
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kSmemOptIn - fa.sharedSizeBytes));
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) != cudaSuccess || per < 1) per = 1;
        if (dev < 16) resident[dev].store(sms * per, std::memory_order_relaxed);
        return sms * per;
    }
};

}  // namespace ld
