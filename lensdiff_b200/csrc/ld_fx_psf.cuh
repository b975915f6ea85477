// ld_fx_psf.cuh — the |FFT|^2 windows of a PSF bank on compiled three-stage
// transforms (ld_fxpass.cuh): the row pass over the pupil's rows and the column
// pass over the window's columns (see psf_rows_kernel and psf_cols_kernel,
// whose work they do).  The pupil is embedded at index 0 instead of the PSF's
// middle: that multiplies the spectrum by phases, which |.|^2 drops, and leaves
// the inputs past the pupil zero, so that the first stage's butterflies have
// their first NZ inputs only (S >= 2 N_p: half of them, a quarter when
// S >= 4 N_p).  Included by the translation units that instantiate the plans'
// kernels (ld_fx_psf*.cu).
#pragma once

#include "ld_fxpass.cuh"

namespace ld {
namespace {

constexpr int psf_seqs(int n) { return n <= 2304 ? 4 : 2; }  // sequences per CTA

// Shared memory: the first stage's outputs lie in blocks of R1 butterfly
// values with one value of padding per sequence after each (its stores, R1
// apart, spread over the banks).
template <class P, int C>
constexpr size_t psf_bytes() {
    return static_cast<size_t>(P::n + P::n / P::R1) * C * sizeof(float2);
}

struct PsfShape {
    int threads, ctas;
};
// As rows_shape: the most useful element slots in flight per SM.
template <class P, int C>
constexpr PsfShape psf_shape() {
    PsfShape best{0, 0};
    double score = -1.0;
    for (int t = 64; t <= 1024; t += 32) {
        const int va = (P::n / P::R1 * C + t - 1) / t * P::R1, vb = (P::n / P::R2 * C + t - 1) / t * P::R2;
        const int vc = (P::n / P::R3 * C + t - 1) / t * P::R3;
        const int v = va > vb ? (va > vc ? va : vc) : (vb > vc ? vb : vc);
        if (v > 32) continue;
        int ctas = static_cast<int>((228 * 1024) / (psf_bytes<P, C>() + 1024));
        if (ctas > 16) ctas = 16;
        while (ctas > 0 && 65536 / ((ctas * t / 32 + 3) / 4 * 128) / 8 * 8 < 2 * v + 24) --ctas;
        if (ctas < 1) continue;
        const double s = 3.0 * P::n * C / (va + vb + vc) * ctas;
        if (s > score) {
            score = s;
            best = PsfShape{t, ctas};
        }
    }
    return best;
}

// A DFT of radix 4 B whose inputs r >= NZ (B or 2 B) are zero: the inner
// radix-4 transforms over r1 (r = B r1 + r2) have one or two inputs.
template <int B, int NZ, int R2, int... K1>
__device__ __forceinline__ void head_col(float2* v, std::integer_sequence<int, K1...>) {
    constexpr int R = 4 * B;
    float2 t[4];
    const float2 a = v[R2];
    if constexpr (NZ == B) {
        t[0] = t[1] = t[2] = t[3] = a;
    } else {
        const float2 b = v[B + R2];
        t[0] = cadd(a, b);
        t[1] = make_float2(a.x + b.y, a.y - b.x);
        t[2] = csub(a, b);
        t[3] = make_float2(a.x - b.y, a.y + b.x);
    }
    ((v[B * K1 + R2] = rotate<R, R2 * K1, false>(t[K1])), ...);
}
template <int B, int NZ, int... R2>
__device__ __forceinline__ void head_cols(float2* v, std::integer_sequence<int, R2...>) {
    (head_col<B, NZ, R2>(v, std::make_integer_sequence<int, 4>{}), ...);
}
template <int R, int NZ>
__device__ __forceinline__ void dft_head(float2* v) {
    constexpr int B = R / 4;
    static_assert(R % 4 == 0 && (NZ == B || NZ == 2 * B));
    head_cols<B, NZ>(v, std::make_integer_sequence<int, B>{});
    float2 o[R];
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
        float2 t[B];
#pragma unroll
        for (int r2 = 0; r2 < B; ++r2) t[r2] = v[B * k1 + r2];
        fdft<B, false>(t);
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) o[k1 + 4 * k2] = t[k2];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = o[r];
}

// First stage: ld(e) for the first NZ inputs of each butterfly; SYNC as fp_stage.
template <class P, int C, int T, int NZ, bool SYNC, class Ld>
__device__ __forceinline__ void psf_first(float2* s, Ld ld) {
    constexpr int R = P::R1, NB = P::n / R * C;
    constexpr int IT = (NB + T - 1) / T;
    const int tid = static_cast<int>(threadIdx.x);
    float2 v[IT][R];
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int b = tid + it * T;
        if ((it + 1) * T <= NB || b < NB) {
#pragma unroll
            for (int r = 0; r < NZ; ++r) v[it][r] = ld(b + r * NB);
        }
    }
    if constexpr (SYNC) __syncthreads();
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int b = tid + it * T;
        if ((it + 1) * T <= NB || b < NB) {
            dft_head<R, NZ>(v[it]);
            const int j = b / C;
            const int base = j * (R + 1) * C + (b - j * C);
#pragma unroll
            for (int r = 0; r < R; ++r) s[base + r * C] = v[it][r];
        }
    }
}

// The second and third stage over the padded first-stage outputs in s.
template <class P, int C, int T, class Last>
__device__ __forceinline__ void psf_rest(float2* s, const float2* stw, Last& last) {
    constexpr int block = P::R1 * C;
    fp_stage<P::n, C, T, false, P::R2, P::R1, true>(
        stw + P::tab2, [&](int e) { return s[e + e / block * C]; }, [&](int e, float2 v) { s[e] = v; });
    __syncthreads();
    last.run(stw + P::tab3, [&](int e) { return s[e]; });
}

// Window coordinate of spectrum index k: the window's pixel w is spectrum index
// (x0 + w + half) mod S.
__device__ __forceinline__ int window_index(int k, int x0, int half, int S) {
    int w = k - half - x0;
    if (w < 0) w += S;
    return w < 0 ? w + S : w;
}

// grid (ceil(row_n / C), B): C pupil rows of wavelength blockIdx.y.  440 rows of
// 2048 for 31 wavelengths take 87 us (266 with the runtime-planned transforms),
// bound by issue: the fields' sine and cosine and the transform.
template <class P, int C, int NZ, int T, int MINB>
__global__ void __launch_bounds__(T, MINB) fx_psf_rows_kernel(PsfBankArgs a) {
    stream_order();
    extern __shared__ __align__(128) unsigned char smraw[];
    constexpr int S = P::n;
    float2* s = reinterpret_cast<float2*>(smraw);
    const int b = blockIdx.y, yr0 = blockIdx.x * C;
    const WavelengthInfo* w = a.wl + b;
    const int np = a.pupil.size;
    const int enabled = w->phase.enabled;
    const float c4 = w->phase.c[4];
    constexpr int filled = S / P::R1 * NZ;  // inputs the first stage reads
#pragma unroll 1
    for (int r = 0; r < C; ++r) {
        const bool row = yr0 + r < a.row_n;
        const float4* pre = a.pupil_pre + static_cast<size_t>(a.row_lo + yr0 + r) * np;
        for (int x = threadIdx.x; x < filled; x += T) {
            float2 f = make_float2(0.0f, 0.0f);
            if (row && x < np) {
                const float4 q = __ldg(pre + x);
                const float ph = (enabled && q.w != 0.0f) ? q.y + c4 * q.z : 0.0f;
                if (!(q.x <= 0.0f)) {
                    float sn, cs;
                    sincosf(ph * 2.0f * kPiF, &sn, &cs);
                    f = make_float2(q.x * cs, q.x * sn);
                }
            }
            s[x * C + r] = f;
        }
    }
    __syncthreads();
    psf_first<P, C, T, NZ, true>(s, [&](int e) { return s[e]; });
    __syncthreads();
    LastStage<S, C, T, false, P::R3> last;
    psf_rest<P, C, T>(s, a.plan_s.stw, last);
    const int wn = w->win_n, x0 = w->win_x0, half = a.half;
    float2* out = a.rows + (static_cast<size_t>(b) * a.row_n + yr0) * a.win_stride;
    const int rows = min(C, a.row_n - yr0);
    last.each([&](int e, float2 v) {
        const int k = e / C, r = e - k * C;
        const int wx = window_index(k, x0, half, S);
        if (wx < wn && r < rows) out[r * a.win_stride + wx] = v;
    });
}

// grid (ceil(win_stride / C), B): C window columns of wavelength blockIdx.y.
// Windows of 236-413 columns of 2048 for 31 wavelengths take 56 us (215).
template <class P, int C, int NZ, int T, int MINB>
__global__ void __launch_bounds__(T, MINB) fx_psf_cols_kernel(PsfBankArgs a) {
    stream_order();
    extern __shared__ __align__(128) unsigned char smraw[];
    constexpr int S = P::n;
    float2* s = reinterpret_cast<float2*>(smraw);
    const int b = blockIdx.y;
    const WavelengthInfo* w = a.wl + b;
    const int wn = w->win_n;
    const int X0 = blockIdx.x * C;
    if (X0 >= wn) return;
    const int rn = a.row_n, stride = a.win_stride;
    const float2* in = a.rows + static_cast<size_t>(b) * rn * stride + X0;
    const int cols = min(C, wn - X0);
    psf_first<P, C, T, NZ, false>(s, [&](int e) {
        const int g = e / C, c = e - g * C;
        return g < rn && c < cols ? __ldg(in + g * stride + c) : make_float2(0.0f, 0.0f);
    });
    __syncthreads();
    LastStage<S, C, T, false, P::R3> last;
    psf_rest<P, C, T>(s, a.plan_s.stw, last);
    const int x0 = w->win_x0, half = a.half;
    float* out = a.win + static_cast<size_t>(b) * stride * stride + X0;
    last.each([&](int e, float2 f) {
        const int k = e / C, c = e - k * C;
        const int wy = window_index(k, x0, half, S);
        if (wy < wn && c < cols) out[static_cast<size_t>(wy) * stride + c] = f.x * f.x + f.y * f.y;
    });
}

template <class P, int NZ>
void psf_launch(const PsfBankArgs& a, bool rows, cudaStream_t s) {
    constexpr int C = psf_seqs(P::n);
    constexpr PsfShape sh = psf_shape<P, C>();
    static_assert(sh.threads > 0);
    constexpr size_t sm = psf_bytes<P, C>();
    if (rows) {
        static KernelState state;
        auto f = fx_psf_rows_kernel<P, C, NZ, sh.threads, sh.ctas>;
        state.get(f, sh.threads, sm);
        launch_after(f, dim3((a.row_n + C - 1) / C, a.B), sh.threads, sm, s, a);
    } else {
        static KernelState state;
        auto f = fx_psf_cols_kernel<P, C, NZ, sh.threads, sh.ctas>;
        state.get(f, sh.threads, sm);
        launch_after(f, dim3((a.win_stride + C - 1) / C, a.B), sh.threads, sm, s, a);
    }
}

// The row (rows) or column pass of plan P; false when the pupil does not fit
// half of S.
template <class P>
bool psf_pass(const PsfBankArgs& a, bool rows, cudaStream_t s) {
    const int np = a.pupil.size;
    if (2 * np > P::n) return false;
    if (4 * np <= P::n) psf_launch<P, P::R1 / 4>(a, rows, s);
    else psf_launch<P, P::R1 / 2>(a, rows, s);
    return true;
}

}  // namespace
}  // namespace ld
