// ld_fx_cols.cuh — the column passes on compiled three-stage transforms
// (ld_fxpass.cuh): the frame's (forward, spectral multiply, inverse) and the
// kernel spectra's.  Included by the translation units that instantiate the
// plans' kernels (ld_fx_cols*.cu).
#pragma once

#include "ld_frame_kernels.cuh"
#include "ld_fxpass.cuh"

namespace ld {
namespace {

// Bytes ahead of a column pass's data: mbarriers and the warps' maxima.
constexpr int kColsHeader = 256;
struct ColsHeader {
    uint64_t bar[3];
    float part[32];
};

// Shared memory of a column pass: C interleaved sequences and one more.
constexpr size_t cols_bytes(int n, int C) { return kColsHeader + static_cast<size_t>(n) * (C + 1) * sizeof(float2); }

// Threads of a column pass over C interleaved sequences: the multiple of 32
// with the most useful element slots in flight per SM.  A stage of radix
// R keeps ceil(C n / R / T) butterflies of R values per thread in registers
// (at most 32 values); a thread needs 80 registers, and each CTA its share of
// shared memory (cols_bytes).  ORD: the FP16 form's passes.
struct ColsShape {
    int threads, ctas;
};
template <class P, int C, bool ORD>
constexpr ColsShape cols_shape() {
    const int radix[4] = {ORD ? P::ord.radix(0) : P::R1, ORD ? P::ord.radix(1) : P::R2,
                          ORD ? P::ord.radix(2) : P::R3, ORD ? P::ord.radix(3) : 0};
    const int count = ORD ? P::ord.count : 3;
    ColsShape best{0, 0};
    double score = -1.0;
    for (int t = 32; t <= 800; t += 32) {
        int steps = 0;
        bool fits = true;
        for (int i = 0; i < count; ++i) {
            const int it = (C * P::n / radix[i] + t - 1) / t;
            steps += it * radix[i];
            if (it * radix[i] > 32) fits = false;
        }
        const int by_smem = static_cast<int>((228 * 1024) / (cols_bytes(P::n, C) + 1024));
        const int by_regs = 65536 / (80 * t);
        int ctas = by_smem < by_regs ? by_smem : by_regs;
        if (ctas > 8) ctas = 8;
        if (!fits || ctas < 1) continue;
        const double s = static_cast<double>(count) * C * P::n / steps * ctas;  // useful slots per SM
        if (s > score) {
            score = s;
            best = ColsShape{t, ctas};
        }
    }
    return best;
}

// The forward passes of the column's order from I on, over the column in F
// (pass 1 on) and the free half of W in turn (one barrier a pass), ending in
// F; an even number of passes takes the first of them in place.
template <class P, int T, int I>
__device__ __forceinline__ void ord_column(const float2* __restrict__ tw, float2* F, float2* W) {
    if constexpr (I < P::ord.count) {
        constexpr bool left_even = (P::ord.count - I) % 2 == 0;
        constexpr bool in_place = !left_even && I == 1;
        const float2* from = left_even || in_place ? F : W;
        float2* to = left_even ? W : F;
        ord_pass<P, 1, T, false, I, in_place>(
            tw, [&](int e) { return from[e]; }, [&](int e, float2 v) { to[e] = v; });
        if constexpr (I + 1 < P::ord.count) __syncthreads();
        ord_column<P, T, I + 1>(tw, F, W);
    }
}

// The last pass of a column transform (H16: of the FP16 form's order).
template <class P, int C, int T, bool INV, bool H16>
struct ColsLastOf {
    using type = LastStage<P::n, C, T, INV, P::R3>;
};
template <class P, int C, int T, bool INV>
struct ColsLastOf<P, C, T, INV, true> {
    using type = OrdLast<P, C, T, INV>;
};
template <class P, int C, int T, bool INV, bool H16>
using ColsLast = typename ColsLastOf<P, C, T, INV, H16>::type;

// Column k = blockIdx.x: its row spectra transformed, multiplied by its C (3 or,
// with the luma lock, 4) kernel spectra, the products transformed back, the
// first Hp rows stored to B.  Shared memory: the header, F [n] (the column's
// spectrum), W [n][C].
// H16 (the passes of P::ord): the half2 row spectra and their row exponents
// arrive at the start of W (widened as the forward transform's first pass
// loads them), the half2 kernel spectra in W's upper half (scaled and
// multiplied with F as the inverse's first pass loads them); the forward
// passes alternate between F and W's lower half, so they need one barrier
// each.  FP32: the row spectra arrive in F, the kernel spectra fill W.  The
// inverse's last pass stays in registers: its largest component (H16: the
// column's scale) and the store come from there.
// Bound by the latency of its passes: at n = 3200, 24 warps per SM of which the
// forward passes (a third of the inverse's butterflies) use some, 51 % of the
// issue slots.  H16 / FP32 launch times, against the passes before it
// (compiled transforms in place between a fill, a product and a drain; at the
// other lengths the runtime-planned transforms):
//   2501 columns of 3200: 140 us (175) / 130 us (155)
//   4097 columns of 5120: 479 us (757; four passes) / 391 us
//   1126 columns of 1800: 43 us H16 (101)
//   1251 columns of 1600: 37 us (50) / 39 us
//   1201 columns of 1152: 29 us FP32 (72)
template <class P, int C, int T, int MINB, bool H16>
__global__ void __launch_bounds__(T, MINB) fx_frame_cols_kernel(FrameArgs a) {
    stream_order();
    extern __shared__ __align__(128) unsigned char smraw[];
    constexpr int N = P::n;
    ColsHeader* h = reinterpret_cast<ColsHeader*>(smraw);
    float2* F = reinterpret_cast<float2*>(smraw + kColsHeader);
    float2* W = F + N;
    const int Hp = a.Hp, cols = a.g.cols;
    const int k = blockIdx.x;
    const uint32_t a_bytes = static_cast<uint32_t>(Hp * (H16 ? sizeof(__half2) : sizeof(float2)));
    constexpr uint32_t k_bytes = static_cast<uint32_t>(N * C * (H16 ? sizeof(__half2) : sizeof(float2)));
    const char* asrc = reinterpret_cast<const char*>(a.A) + static_cast<size_t>(k) * a_bytes;
    const char* ksrc = reinterpret_cast<const char*>(a.spectra) + static_cast<size_t>(k) * k_bytes;
    __half2* ah = reinterpret_cast<__half2*>(W);
    signed char* aex = reinterpret_cast<signed char*>(ah + Hp);
    __half2* kh = reinterpret_cast<__half2*>(W) + C * N;
    if (threadIdx.x == 0) {
        mbar_init(&h->bar[0], 1);
        mbar_init(&h->bar[1], 1);
        if (H16) mbar_init(&h->bar[2], 1);
        mbar_init_fence();
        bulk_load_checked(H16 ? static_cast<void*>(ah) : static_cast<void*>(F), asrc, a_bytes, &h->bar[0], smraw, a.err);
        if (H16)
            bulk_load_checked(aex, a.aexp, static_cast<uint32_t>((Hp + 15) & ~15), &h->bar[2], smraw, a.err);
        bulk_load_checked(H16 ? static_cast<void*>(kh) : static_cast<void*>(W), ksrc, k_bytes, &h->bar[1], smraw, a.err);
        const int later = k + a.ahead;
        if (later < cols) {
            bulk_prefetch_l2(asrc + static_cast<size_t>(later - k) * a_bytes, a_bytes);
            bulk_prefetch_l2(ksrc + static_cast<size_t>(later - k) * k_bytes, k_bytes);
        }
    }
    __syncthreads();  // barriers initialised before anyone waits on them
    const float2* tw = a.g.plan_py.stw;
    if (__syncthreads_or(!mbar_wait(&h->bar[0], 0, a.err) || (H16 && !mbar_wait(&h->bar[2], 0, a.err)))) return;
    auto ldF = [&](int e) { return F[e]; };
    auto stF = [&](int e, float2 v) { F[e] = v; };
    auto ldW = [&](int e) { return W[e]; };
    auto stW = [&](int e, float2 v) { W[e] = v; };
    const float2 zero = make_float2(0.0f, 0.0f);
    if constexpr (H16) {
        const float2* otw = ord_table<P, C == 3>(tw);
        ord_pass<P, 1, T, false, 0, false>(
            otw, [&](int e) { return e < Hp ? from_half2(ah[e], exp2_int(aex[e])) : zero; }, stF);
        __syncthreads();
        ord_column<P, T, 1>(otw, F, W);
    } else {
        fp_stage<N, 1, T, false, P::R1, 1, true>(nullptr, [&](int e) { return e < Hp ? F[e] : zero; }, stF);
        __syncthreads();
        fp_stage<N, 1, T, false, P::R2, P::R1, true>(tw + P::tab2, ldF, stF);
        __syncthreads();
        fp_stage<N, 1, T, false, P::R3, P::R1 * P::R2, true>(tw + P::tab3, ldF, stF);
    }
    if (__syncthreads_or(!mbar_wait(&h->bar[1], 0, a.err))) return;
    ColsLast<P, C, T, true, H16> last;
    if constexpr (H16) {
        const float2* otw = ord_table<P, C == 3>(tw);
        const float ks = a.kscale[k];
        ord_pass<P, C, T, true, 0, true>(otw, [&](int e) { return cmul(from_half2(kh[e], ks), F[e / C]); }, stW);
        __syncthreads();
        ord_middle<P, C, T, true>(otw, W);
        last.run(otw + P::ord.table(P::ord.count - 1), ldW);
    } else {
        fp_stage<N, C, T, true, P::R1, 1, true>(nullptr, [&](int e) { return cmul(W[e], F[e / C]); }, stW);
        __syncthreads();
        fp_stage<N, C, T, true, P::R2, P::R1, true>(tw + P::tab2, ldW, stW);
        __syncthreads();
        last.run(tw + P::tab3, ldW);
    }
    // element e = row * C + c of column k goes to B's group of four columns
    const int64_t base = (static_cast<int64_t>(k / kBGroup) * Hp * kBGroup + k % kBGroup) * C;
    constexpr int step = kBGroup * C;
    if constexpr (H16) {
        float m = 0.0f;
        last.each([&](int e, float2 v) {
            if (e < Hp * C) m = fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y)));
        });
        m = cta_max<T>(m, h->part);
        const float sc = m > 0.0f ? kHalfTop / m : 1.0f;
        if (threadIdx.x == 0) a.bscale[k] = m > 0.0f ? m / kHalfTop : 1.0f;
        __half2* out = reinterpret_cast<__half2*>(a.Bout) + base;
        last.each([&](int e, float2 v) {
            const int row = e / C;
            if (row < Hp) out[row * step + (e - row * C)] = to_half2(v, sc);
        });
    } else {
        float2* out = a.Bout + base;
        last.each([&](int e, float2 v) {
            const int row = e / C;
            if (row < Hp) out[row * step + (e - row * C)] = v;
        });
    }
}

// The Mono column pass (FP32): the three colours' row spectra (X [n][3], arriving
// in its first Hp rows) transformed, multiplied by the one kernel spectrum
// (Kc [n]), transformed back.  321 columns of 400 take 7.8 us (16.8 with the
// runtime-planned transforms), the scatter's 1001 of 1200 35 us (60).
template <class P, int T, int MINB>
__global__ void __launch_bounds__(T, MINB) fx_frame_cols_mono_kernel(FrameArgs a) {
    stream_order();
    extern __shared__ __align__(128) unsigned char smraw[];
    constexpr int N = P::n, C = 3;
    ColsHeader* h = reinterpret_cast<ColsHeader*>(smraw);
    float2* X = reinterpret_cast<float2*>(smraw + kColsHeader);
    float2* Kc = X + C * N;
    const int Hp = a.Hp, cols = a.g.cols;
    const int k = blockIdx.x;
    const uint32_t a_bytes = static_cast<uint32_t>(Hp * C * sizeof(float2));
    constexpr uint32_t k_bytes = N * sizeof(float2);
    const float2* asrc = a.A + static_cast<size_t>(k) * Hp * C;
    const float2* ksrc = a.spectra + static_cast<size_t>(k) * N;
    if (threadIdx.x == 0) {
        mbar_init(&h->bar[0], 1);
        mbar_init(&h->bar[1], 1);
        mbar_init_fence();
        bulk_load_checked(X, asrc, a_bytes, &h->bar[0], smraw, a.err);
        bulk_load_checked(Kc, ksrc, k_bytes, &h->bar[1], smraw, a.err);
        const int later = k + a.ahead;
        if (later < cols) {
            bulk_prefetch_l2(a.A + static_cast<size_t>(later) * Hp * C, a_bytes);
            bulk_prefetch_l2(a.spectra + static_cast<size_t>(later) * N, k_bytes);
        }
    }
    __syncthreads();  // barriers initialised before anyone waits on them
    const float2* tw = a.g.plan_py.stw;
    if (__syncthreads_or(!mbar_wait(&h->bar[0], 0, a.err))) return;
    auto ld = [&](int e) { return X[e]; };
    auto st = [&](int e, float2 v) { X[e] = v; };
    fp_stage<N, C, T, false, P::R1, 1, true>(
        nullptr, [&](int e) { return e < Hp * C ? X[e] : make_float2(0.0f, 0.0f); }, st);
    __syncthreads();
    fp_stage<N, C, T, false, P::R2, P::R1, true>(tw + P::tab2, ld, st);
    __syncthreads();
    fp_stage<N, C, T, false, P::R3, P::R1 * P::R2, true>(tw + P::tab3, ld, st);
    if (__syncthreads_or(!mbar_wait(&h->bar[1], 0, a.err))) return;
    fp_stage<N, C, T, true, P::R1, 1, true>(nullptr, [&](int e) { return cmul(X[e], Kc[e / C]); }, st);
    __syncthreads();
    fp_stage<N, C, T, true, P::R2, P::R1, true>(tw + P::tab2, ld, st);
    __syncthreads();
    LastStage<N, C, T, true, P::R3> last;
    last.run(tw + P::tab3, ld);
    float2* out = a.Bout + (static_cast<int64_t>(k / kBGroup) * Hp * kBGroup + k % kBGroup) * C;
    last.each([&](int e, float2 v) {
        const int row = e / C;
        if (row < Hp) out[row * (kBGroup * C) + (e - row * C)] = v;
    });
}

// Column k of the C kernel spectra: the row spectra of the canvas rows (Kp x C)
// arrive by bulk copy behind W, take their wrapped grid rows as the first
// stage loads them, and the last stage's registers go out to KS[k] (H16: in
// FP16 with the column's scale).  H16 / FP32: 2501 columns of 3200 take 89 / 90
// us (128 before, see above), 4097 of 5120 331 / 289 us (517), 1126 of 1800 28
// us H16 (66).
template <class P, int C, int T, int MINB, bool H16>
__global__ void __launch_bounds__(T, MINB) fx_kspec_cols_kernel(KernelSpectraArgs a) {
    stream_order();
    extern __shared__ __align__(128) unsigned char smraw[];
    constexpr int N = P::n;
    ColsHeader* h = reinterpret_cast<ColsHeader*>(smraw);
    float2* W = reinterpret_cast<float2*>(smraw + kColsHeader);
    float2* Rb = W + C * N;
    const int cols = a.g.cols, Kp = a.Kp, R = a.R;
    const int k = blockIdx.x;
    const uint32_t r_bytes = static_cast<uint32_t>(Kp * C * sizeof(float2));
    if (threadIdx.x == 0) {
        mbar_init(&h->bar[0], 1);
        mbar_init_fence();
        bulk_load_checked(Rb, a.rows + static_cast<size_t>(k) * Kp * C, r_bytes, &h->bar[0], smraw, a.err);
        const int later = k + a.ahead;
        if (later < cols) bulk_prefetch_l2(a.rows + static_cast<size_t>(later) * Kp * C, r_bytes);
    }
    __syncthreads();  // barrier initialised before anyone waits on it
    const float2* tw = a.g.plan_py.stw;
    if (__syncthreads_or(!mbar_wait(&h->bar[0], 0, a.err))) return;
    auto ldW = [&](int e) { return W[e]; };
    auto stW = [&](int e, float2 v) { W[e] = v; };
    // grid row v holds canvas row v + R (v <= R) or v - N + R (v >= N - R)
    auto ldR = [&](int e) {
        const int lo = e + C * R, hi = e - C * (N - R);
        if (e < C * (R + 1)) return Rb[lo];
        if (hi >= 0) return Rb[hi];
        return make_float2(0.0f, 0.0f);
    };
    ColsLast<P, C, T, false, H16> last;
    if constexpr (H16) {
        const float2* otw = ord_table<P, C == 3>(tw);
        const float scale = a.scale;
        ord_pass<P, C, T, false, 0, false>(otw, [&](int e) { return cscale(ldR(e), scale); }, stW);
        __syncthreads();
        ord_middle<P, C, T, false>(otw, W);
        last.run(otw + P::ord.table(P::ord.count - 1), ldW);
    } else {
        fp_stage<N, C, T, false, P::R1, 1, false>(nullptr, ldR, stW);
        __syncthreads();
        fp_stage<N, C, T, false, P::R2, P::R1, true>(tw + P::tab2, ldW, stW);
        __syncthreads();
        last.run(tw + P::tab3, ldW);
    }
    if constexpr (H16) {
        float m = 0.0f;
        last.each([&](int, float2 v) { m = fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))); });
        m = cta_max<T>(m, h->part);
        const float sc = m > 0.0f ? kHalfTop / m : 1.0f;
        if (threadIdx.x == 0) a.kscale[k] = m > 0.0f ? m / kHalfTop : 1.0f;
        __half2* out = reinterpret_cast<__half2*>(a.spectra) + static_cast<size_t>(k) * N * C;
        last.each([&](int e, float2 v) { out[e] = to_half2(v, sc); });
    } else {
        float2* out = a.spectra + static_cast<size_t>(k) * N * C;
        const float sc = a.scale;
        last.each([&](int e, float2 v) { out[e] = cscale(v, sc); });
    }
}

template <class P, int C, bool H16>
void frame_cols_fx(FrameArgs a, cudaStream_t s) {
    constexpr ColsShape sh = cols_shape<P, C, H16>();
    static_assert(sh.threads > 0);
    static KernelState state;
    auto f = fx_frame_cols_kernel<P, C, sh.threads, sh.ctas, H16>;
    constexpr size_t sm = cols_bytes(P::n, C);
    a.ahead = state.get(f, sh.threads, sm);
    if (a.g.cols > 0) launch_after(f, a.g.cols, sh.threads, sm, s, a);  // (none: to load the kernel)
}

template <class P>
void frame_cols_mono_fx(FrameArgs a, cudaStream_t s) {
    constexpr ColsShape sh = cols_shape<P, 3, false>();
    static KernelState state;
    auto f = fx_frame_cols_mono_kernel<P, sh.threads, sh.ctas>;
    constexpr size_t sm = cols_bytes(P::n, 3);
    a.ahead = state.get(f, sh.threads, sm);
    launch_after(f, a.g.cols, sh.threads, sm, s, a);
}

template <class P, int C, bool H16>
bool kspec_cols_fx(KernelSpectraArgs a, cudaStream_t s) {
    constexpr ColsShape sh = cols_shape<P, C, H16>();
    static_assert(sh.threads > 0);
    static KernelState state;
    auto f = fx_kspec_cols_kernel<P, C, sh.threads, sh.ctas, H16>;
    const size_t sm = kColsHeader + (static_cast<size_t>(P::n) + a.Kp) * C * sizeof(float2);
    if (sm > kSmemOptIn) return false;
    a.ahead = state.get(f, sh.threads, cols_bytes(P::n, C));
    if (a.g.cols > 0) launch_after(f, a.g.cols, sh.threads, sm, s, a);
    return true;
}

// The FP16 form's launch, where the plan has an order.
template <class P, int C>
bool cols_launch_h16(const FrameArgs* fa, const KernelSpectraArgs* ka, cudaStream_t s) {
    if constexpr (P::ord.count > 0) {
        if (ka) return kspec_cols_fx<P, C, true>(*ka, s);
        frame_cols_fx<P, C, true>(*fa, s);
        return true;
    }
    return false;
}

// The launch of plan P: the frame's column pass (fa) or the kernel spectra's
// (ka); false when it does not fit, for the Mono and luma-lock chains at
// lengths above kFxOtherMax, and in the FP16 form where the plan has no order:
// those stay on the runtime-planned transforms.
template <class P>
bool cols_launch(const FrameArgs* fa, const KernelSpectraArgs* ka, cudaStream_t s) {
    const bool h16 = fa ? fa->h16 != 0 : ka->h16 != 0;
    if (fa ? fa->n_drv == 1 && fa->n_out == 3 : ka->n_ker == 3) {
        if (h16) return cols_launch_h16<P, 3>(fa, ka, s);
        if (ka) return kspec_cols_fx<P, 3, false>(*ka, s);
        frame_cols_fx<P, 3, false>(*fa, s);
        return true;
    }
    if constexpr (P::n <= kFxOtherMax) {
        if (fa && fa->n_drv == 3) {
            frame_cols_mono_fx<P>(*fa, s);
            return true;
        }
        if (ka && ka->n_ker == 1) return kspec_cols_fx<P, 1, false>(*ka, s);
        if (h16) return cols_launch_h16<P, 4>(fa, ka, s);
        if (ka) return kspec_cols_fx<P, 4, false>(*ka, s);
        frame_cols_fx<P, 4, false>(*fa, s);
        return true;
    }
    return false;
}

}  // namespace
}  // namespace ld
