// ld_fx_rows.cuh — the row passes on compiled three-stage transforms
// (ld_fxpass.cuh): the frame's forward rows (with the highlight extraction),
// its inverse rows (with the composite) and the kernel spectra's rows.  The
// real rows of length 2M run as complex transforms of length M; bin k of the
// real transform needs Z[k] and Z[M - k], which lie in the mirrored
// butterflies p and M/R - p of a stage of radix R that spans the row (the
// forward transform's last, the inverse's first).  A thread therefore takes
// both butterflies and forms the bins, or the complex row, in registers.
// Included by the translation units that instantiate the plans' kernels
// (ld_fx_rows*.cu).
#pragma once

#include "ld_frame_kernels.cuh"
#include "ld_fxpass.cuh"

namespace ld {
namespace {

constexpr int kRowsHeader = 128;  // the warps' maxima (at most 32 floats)

// A row plan: forward radices R1, R2, R3, the inverse in reverse; ord: the FP16
// form's forward order.  Stage tables: the forward radices' second and third
// stage, then the inverse's, then the order's.
template <int R1_, int R2_, int R3_>
struct FxRow {
    static constexpr int R1 = R1_, R2 = R2_, R3 = R3_;
    static constexpr int n = R1 * R2 * R3;
    static constexpr int tab2 = 0, tab3 = R1 * FxPad<R2>::value;
    static constexpr int inv2 = tab3 + R1 * R2 * FxPad<R3>::value;
    static constexpr int inv3 = inv2 + R3 * FxPad<R2>::value;
    static constexpr int tab_ord = inv3 + R3 * R2 * FxPad<R1>::value;
    static constexpr FxOrder ord = fx_row_order(R1, R2, R3);  // count 0: none
    static constexpr bool table_twiddles = fx_table_twiddles(true, n);
};

// Threads and CTAs per SM of a row pass over C sequences whose mirrored stage
// has radix RM and whose others have RA, RB and (0: none) RC: the multiple of
// 32 with the most useful element slots in flight per SM.  A thread holding
// up to v values (at most 32) needs 2 v + 24 registers; an SM gives registers
// to warps four at a time.
struct RowsShape {
    int threads, ctas;
};
constexpr RowsShape rows_shape(int n, int C, int RA, int RB, int RC, int RM) {
    RowsShape best{0, 0};
    double score = -1.0;
    const int others[3] = {RA, RB, RC};
    for (int t = 32; t <= 1024; t += 32) {
        int v = ((n / RM / 2 + 1) * C + t - 1) / t * 2 * RM, sum = v, stages = 1;
        for (int r : others) {
            if (r == 0) continue;
            const int vr = (n / r * C + t - 1) / t * r;
            v = vr > v ? vr : v;
            sum += vr;
            ++stages;
        }
        if (v > 32) continue;
        int ctas = static_cast<int>((228 * 1024) / (kRowsHeader + n * C * 8 + 1024));
        if (ctas > 16) ctas = 16;
        while (ctas > 0 && 65536 / ((ctas * t / 32 + 3) / 4 * 128) / 8 * 8 < 2 * v + 24) --ctas;
        if (ctas < 1) continue;
        const double s = static_cast<double>(stages) * n * C / sum * ctas;
        if (s > score) {
            score = s;
            best = RowsShape{t, ctas};
        }
    }
    return best;
}
template <class P, int C>
constexpr RowsShape ord_rows_shape() {
    return rows_shape(P::n, C, P::ord.radix(0), P::ord.count > 2 ? P::ord.radix(1) : 0,
                      P::ord.count > 3 ? P::ord.radix(2) : 0, P::ord.radix(P::ord.count - 1));
}

// The mirrored butterflies p and Q - p (Q = N / R) of a stage: a[it] and b[it]
// of task t = tid + it * T, p = t / C in [0, Q / 2], sequence t % C.
template <int N, int C, int T, int R, class Stage = FastStage>
struct Mirror {
    static constexpr int Q = N / R;
    static constexpr int TASKS = (Q / 2 + 1) * C;
    static constexpr int IT = (TASKS + T - 1) / T;
    float2 a[IT][R], b[IT][R];
    static __device__ __forceinline__ int task(int it) { return static_cast<int>(threadIdx.x) + it * T; }
    static __device__ __forceinline__ bool has(int it) { return (it + 1) * T <= TASKS || task(it) < TASKS; }

    // The forward transform's last stage over smem s, then bins k = p + r Q
    // (a[it][r]) and N - k (b[it][R - 1 - r]) of the real transform of length
    // 2N (tw: exp(-2 pi i k / 2N)).
    __device__ __forceinline__ void forward(const float2* s, const float2* __restrict__ stw,
                                            const float2* __restrict__ tw) {
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            if (!has(it)) continue;
            const int p = task(it) / C, c = task(it) - p * C;
            const int q = p == 0 ? 0 : Q - p;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                a[it][r] = s[(p + r * Q) * C + c];
                b[it][r] = s[(q + r * Q) * C + c];
            }
        }
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            if (!has(it)) continue;
            const int p = task(it) / C;
            Stage::template run<false, R, Q>(a[it], p, stw);
            if (p != 0) {
                Stage::template run<false, R, Q>(b[it], Q - p, stw);
            } else {  // Z[N - rQ] = Z[(R - r) Q]
#pragma unroll
                for (int r = 0; r < R; ++r) b[it][r] = a[it][(r + 1) % R];
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float2 zk = a[it][r], zm = b[it][R - 1 - r];
                const float2 w = __ldg(&tw[p + r * Q]);
                const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
                const float2 o = make_float2(0.5f * (zk.y + zm.y), 0.5f * (zm.x - zk.x));
                const float2 t = cmul(w, o);
                a[it][r] = cadd(e, t);
                b[it][R - 1 - r] = make_float2(e.x - t.x, t.y - e.y);
            }
        }
    }
    // f(k, c, value) for every bin the thread holds, each bin once
    template <class F>
    __device__ __forceinline__ void bins(F f) const {
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            if (!has(it)) continue;
            const int p = task(it) / C, c = task(it) - p * C;
#pragma unroll
            for (int r = 0; r < R; ++r) f(p + r * Q, c, a[it][r]);
            if (p != 0 && 2 * p != Q) {
#pragma unroll
                for (int r = 0; r < R; ++r) f(N - (p + r * Q), c, b[it][R - 1 - r]);
            } else if (p == 0) {
                f(N, c, b[it][R - 1]);
            }
        }
    }
    // Largest |component| of the bins
    __device__ __forceinline__ float largest() const {
        float m = 0.0f;
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            if (!has(it)) continue;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                m = fmaxf(m, fmaxf(fabsf(a[it][r].x), fabsf(a[it][r].y)));
                m = fmaxf(m, fmaxf(fabsf(b[it][r].x), fabsf(b[it][r].y)));
            }
        }
        return m;
    }
    // The inverse transform's first stage into smem s: ld(k, c) gives bin k of
    // the real transform, the complex rows' values Z[k], Z[N - k] come from
    // bins k and N - k.
    template <class Ld>
    __device__ __forceinline__ void inverse(float2* s, const float2* __restrict__ tw, Ld ld) {
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            if (!has(it)) continue;
            const int p = task(it) / C, c = task(it) - p * C;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                a[it][r] = ld(p + r * Q, c);
                b[it][R - 1 - r] = ld(N - (p + r * Q), c);
            }
        }
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            if (!has(it)) continue;
            const int p = task(it) / C, c = task(it) - p * C;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float2 xk = a[it][r], xm = b[it][R - 1 - r];
                const float2 w = __ldg(&tw[p + r * Q]);
                const float2 e = make_float2(0.5f * (xk.x + xm.x), 0.5f * (xk.y - xm.y));
                const float2 d = make_float2(0.5f * (xk.x - xm.x), 0.5f * (xk.y + xm.y));
                const float2 o = cmulc(d, w);
                a[it][r] = make_float2(e.x - o.y, e.y + o.x);           // e + i o
                b[it][R - 1 - r] = make_float2(e.x + o.y, o.x - e.y);   // conj(e) + i conj(o)
            }
            fdft<R, true>(a[it]);
#pragma unroll
            for (int r = 0; r < R; ++r) s[(p * R + r) * C + c] = a[it][r];
            if (p != 0 && 2 * p != Q) {
                fdft<R, true>(b[it]);
#pragma unroll
                for (int r = 0; r < R; ++r) s[((Q - p) * R + r) * C + c] = b[it][r];
            }
        }
    }
};

// The mirrored last stage of a forward row pass (H16: of the FP16 form's order).
template <class P, int C, int T, bool H16>
struct RowsLastOf {
    using type = Mirror<P::n, C, T, P::R3>;
};
template <class P, int C, int T>
struct RowsLastOf<P, C, T, true> {
    using type = Mirror<P::n, C, T, P::ord.radix(P::ord.count - 1), OrdStage<P, P::ord.count - 1>>;
};
template <class P, int C, int T, bool H16>
using RowsLast = typename RowsLastOf<P, C, T, H16>::type;

// The forward transform of C rows of smem s: the first stage's inputs from
// ld(e) (IN_PLACE: s itself), the bins left in `last`.  SPECTRAL: see ord_table.
template <class P, int C, int T, bool H16, bool SPECTRAL, bool IN_PLACE, class Ld>
__device__ __forceinline__ void rows_forward(const FftPlan& plan, const float2* __restrict__ tw_px, float2* s,
                                             RowsLast<P, C, T, H16>& last, Ld ld) {
    auto lds = [&](int e) { return s[e]; };
    auto sts = [&](int e, float2 v) { s[e] = v; };
    const float2* stw = plan.stw;
    if constexpr (H16) {
        const float2* otw = ord_table<P, SPECTRAL>(stw);
        ord_pass<P, C, T, false, 0, IN_PLACE>(otw, ld, sts);
        __syncthreads();
        ord_middle<P, C, T, false>(otw, s);
        last.forward(s, otw + P::ord.table(P::ord.count - 1), tw_px);
    } else {
        fp_stage<P::n, C, T, false, P::R1, 1, IN_PLACE>(nullptr, ld, sts);
        __syncthreads();
        fp_stage<P::n, C, T, false, P::R2, P::R1, true>(stw + P::tab2, lds, sts);
        __syncthreads();
        last.forward(s, stw + P::tab3, tw_px);
    }
}

// ---- forward rows ---------------------------------------------------------------
// C / NDRV frame rows per CTA (see frame_rows_kernel, whose work it does): the
// last stage gives the bins, scaled and stored from registers.  Bound by the
// latency of the fill and of the scattered stores (29 % of the warp slots, 40 %
// of the issue slots, the source read once): H16 / FP32, 2160 rows of 2500 take
// 69 / 67 us (88 before: in-place stages and bins through shared memory), 3160
// of 4096 162 / 168 us (207, runtime-planned).  The pixels'
// drivers go through shared memory: forming them in the first stage's
// unrolled loads repeats the highlight mask 50 times and stalls on
// instruction fetches (142 us for 2160 rows of 2500, against 88 before).
template <class P, int C, int NDRV, bool FROM_EFFECT, bool H16, int T, int MINB>
__global__ void __launch_bounds__(T, MINB) fx_frame_rows_kernel(FrameArgs a) {
    stream_order();
    extern __shared__ __align__(128) unsigned char smraw[];
    constexpr int M = P::n;
    float* part = reinterpret_cast<float*>(smraw);
    float2* s = reinterpret_cast<float2*>(smraw + kRowsHeader);
    const int y0 = blockIdx.x * (C / NDRV);
    fill_rows<C, NDRV, FROM_EFFECT>(a, y0, M, s);
    __syncthreads();
    RowsLast<P, C, T, H16> last;
    rows_forward<P, C, T, H16, true, true>(a.g.plan_m, a.g.tw_px, s, last, [&](int e) { return s[e]; });
    const int Hp = a.Hp;
    if constexpr (H16) {
        const int e = row_tile_exp(cta_max<T>(last.largest(), part));
        const float sc = exp2_int(-e);
        if (static_cast<int>(threadIdx.x) < C) a.aexp[y0 + threadIdx.x] = static_cast<signed char>(e);
        __half2* out = reinterpret_cast<__half2*>(a.A) + y0;
        last.bins([&](int k, int c, float2 v) { out[static_cast<int64_t>(k) * Hp + c] = to_half2(v, sc); });
    } else {
        float2* out = a.A + static_cast<int64_t>(y0) * NDRV;
        last.bins([&](int k, int c, float2 v) { out[static_cast<int64_t>(k) * Hp * NDRV + c] = v; });
    }
}

// ---- inverse rows ---------------------------------------------------------------
// One row of C channels per CTA (see frame_inverse_kernel): the first stage
// takes the row's bins from the column outputs, two bins per load pair.  Bound
// by instruction issue and latency (54 % of the issue slots at 24 warps per SM;
// half the instructions are the composite's): H16 / FP32, 2160 rows of 2500 take
// 107 / 110 us (143 / 128 with compiled in-place stages), 3160 of 4096 355 / 439
// us (475 H16, runtime-planned).
template <class P, int C, bool H16, int T, int MINB>
__global__ void __launch_bounds__(T, MINB) fx_frame_inverse_kernel(FrameArgs a) {
    stream_order();
    extern __shared__ __align__(128) unsigned char smraw[];
    constexpr int M = P::n;
    float2* s = reinterpret_cast<float2*>(smraw + kRowsHeader);
    const InverseRow w = inverse_row(a);
    inverse_prefetch(a, w);
    if (w.have) {
        const int Hp = a.Hp, by = w.by;
        const float2* stw = a.g.plan_m.stw;
        {
            Mirror<M, C, T, P::R3> first;
            // b_index in 32 bits: B holds at most 4097 columns of 4 channels
            const int group = Hp * (kBGroup * C);
            const __half2* bh = reinterpret_cast<const __half2*>(a.Bout) + by * (kBGroup * C);
            const float2* bf = a.Bout + by * (kBGroup * C);
            first.inverse(s, a.g.tw_px, [&](int k, int c) {
                const int i = (k >> 2) * group + (k & 3) * C + c;
                if constexpr (H16) return from_half2(__ldcs(bh + i), __ldg(&a.bscale[k]));
                else return __ldcs(bf + i);
            });
        }
        auto ld = [&](int e) { return s[e]; };
        auto st = [&](int e, float2 v) { s[e] = v; };
        __syncthreads();
        fp_stage<M, C, T, true, P::R2, P::R3, true>(stw + P::inv2, ld, st);
        __syncthreads();
        fp_stage<M, C, T, true, P::R1, P::R3 * P::R2, true>(stw + P::inv3, ld, st);
        __syncthreads();
    }
    inverse_epilogue<C>(a, w, s);
}

// ---- kernel-spectrum rows ---------------------------------------------------------
// One canvas row of the C kernels per CTA (see kspec_rows_kernel).  1026 rows of
// 2500 take 54 us (64 before), 1502 of 4096 160 us (214), 1026 of 1125 25 us (75).
template <class P, int C, bool H16, int T, int MINB>
__global__ void __launch_bounds__(T, MINB) fx_kspec_rows_kernel(KernelSpectraArgs a) {
    stream_order();
    extern __shared__ __align__(128) unsigned char smraw[];
    constexpr int M = P::n;
    float2* s = reinterpret_cast<float2*>(smraw + kRowsHeader);
    const int i = blockIdx.x;
    const int R = a.R, K = a.K;
    const size_t kk = static_cast<size_t>(K) * K;
    const float* crow = a.canvas + static_cast<size_t>(i < K ? i : 0) * K;
    const bool zero_row = i >= K;  // the padding row of an odd K
    RowsLast<P, C, T, H16> last;
    rows_forward<P, C, T, H16, C == 3, false>(a.g.plan_m, a.g.tw_px, s, last, [&](int e) {
        const int idx = e / C, c = e - idx * C;
        const float* p = crow + c * kk;
        const int j0 = zero_row ? -1 : canvas_index(2 * idx, 2 * M, R);
        const int j1 = zero_row ? -1 : canvas_index(2 * idx + 1, 2 * M, R);
        return make_float2(j0 >= 0 ? __ldg(p + j0) : 0.0f, j1 >= 0 ? __ldg(p + j1) : 0.0f);
    });
    float2* out = a.rows + static_cast<int64_t>(i) * C;
    const int64_t stride = static_cast<int64_t>(a.Kp) * C;
    last.bins([&](int k, int c, float2 v) { out[k * stride + c] = v; });
}

// Frame rows per CTA of the spectral forward pass: four where they fit the
// shared memory of several CTAs (16-byte runs of A per bin), else two.
constexpr int rows_per_cta(int n) { return n <= 1300 ? 4 : 2; }

template <class P, int C, bool H16>
constexpr RowsShape forward_shape() {
    if constexpr (H16) return ord_rows_shape<P, C>();
    else return rows_shape(P::n, C, P::R1, P::R2, 0, P::R3);
}

template <class P, int C, int NDRV, bool FROM_EFFECT, bool H16 = false>
void frame_rows_fx(const FrameArgs& a, cudaStream_t s) {
    constexpr RowsShape sh = forward_shape<P, C, H16>();
    static_assert(sh.threads > 0);
    static KernelState state;
    auto f = fx_frame_rows_kernel<P, C, NDRV, FROM_EFFECT, H16, sh.threads, sh.ctas>;
    const size_t sm = kRowsHeader + static_cast<size_t>(P::n) * C * sizeof(float2);
    state.get(f, sh.threads, sm);
    launch_after(f, a.Hp / (C / NDRV), sh.threads, sm, s, a);
}

template <class P, int C, bool H16>
void frame_inverse_fx(FrameArgs a, int rows, cudaStream_t s) {
    constexpr RowsShape sh = rows_shape(P::n, C, P::R1, P::R2, 0, P::R3);
    static_assert(sh.threads > 0);
    static KernelState state;
    auto f = fx_frame_inverse_kernel<P, C, H16, sh.threads, sh.ctas>;
    const size_t sm = kRowsHeader + static_cast<size_t>(P::n) * C * sizeof(float2);
    a.ahead = state.get(f, sh.threads, sm);
    launch_after(f, rows, sh.threads, sm, s, a);
}

template <class P, int C, bool H16>
void kspec_rows_fx(const KernelSpectraArgs& a, cudaStream_t s) {
    constexpr RowsShape sh = forward_shape<P, C, H16>();
    static_assert(sh.threads > 0);
    static KernelState state;
    auto f = fx_kspec_rows_kernel<P, C, H16, sh.threads, sh.ctas>;
    const size_t sm = kRowsHeader + static_cast<size_t>(P::n) * C * sizeof(float2);
    state.get(f, sh.threads, sm);
    launch_after(f, a.Kp, sh.threads, sm, s, a);
}

// The launch of plan P named by `pass`; false for the Mono and luma-lock chains
// at lengths above kFxOtherMax, and in the FP16 form where the plan has no order.
template <class P>
bool rows_launch(int pass, const FrameArgs* fa, const KernelSpectraArgs* ka, int rows, cudaStream_t s) {
    constexpr bool other = P::n <= kFxOtherMax, order = P::ord.count > 0;
    if (pass == kFxPassRows) {
        if (fa->n_drv == 1) {
            if (!fa->h16) {
                frame_rows_fx<P, rows_per_cta(P::n), 1, false>(*fa, s);
                return true;
            }
            if constexpr (order) frame_rows_fx<P, rows_per_cta(P::n), 1, false, true>(*fa, s);
            return order;
        }
        if constexpr (other) {
            if (fa->drv_effect) frame_rows_fx<P, 3, 3, true>(*fa, s);
            else frame_rows_fx<P, 3, 3, false>(*fa, s);
            return true;
        }
    } else if (pass == kFxPassInverse) {
        if (fa->n_out == 3) {
            if (fa->h16) frame_inverse_fx<P, 3, true>(*fa, rows, s);
            else frame_inverse_fx<P, 3, false>(*fa, rows, s);
            return true;
        }
        if constexpr (other) {
            if (fa->h16) frame_inverse_fx<P, 4, true>(*fa, rows, s);
            else frame_inverse_fx<P, 4, false>(*fa, rows, s);
            return true;
        }
    } else if (ka->h16) {
        if constexpr (order) {
            if (ka->n_ker == 3) {
                kspec_rows_fx<P, 3, true>(*ka, s);
                return true;
            }
            if constexpr (other) {
                if (ka->n_ker == 4) {
                    kspec_rows_fx<P, 4, true>(*ka, s);
                    return true;
                }
            }
        }
    } else {
        if (ka->n_ker == 3) {
            kspec_rows_fx<P, 3, false>(*ka, s);
            return true;
        }
        if constexpr (other) {
            if (ka->n_ker == 1) kspec_rows_fx<P, 1, false>(*ka, s);
            else kspec_rows_fx<P, 4, false>(*ka, s);
            return true;
        }
    }
    return false;
}

}  // namespace
}  // namespace ld
