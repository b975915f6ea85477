// ld_psf.cu — PSF-bank kernels: pupil -> |FFT|^2 window -> lambda-rescale ->
// kernel shaping -> adaptive crop/taper -> weighted combination.
//
// Reference stages (LensDiffCpuReference.cpp):
//   buildPupilAmplitude / BuildLensDiffPupilPhaseWaves :758-829
//                           -> pupil_pre_kernel (once per bank)
//   buildShiftedRawPsf      :831-859   -> psf_rows_kernel + psf_cols_kernel
//   makeResampledKernel     :1060-1086 -> resample_kernel
//   azimuthalMeanKernel / reshapeAnisotropy / estimateAdaptiveSupportRadius
//                           :1088-1135, :984-1031 -> shape_stats_kernel, support_kernel
//   cropKernelToRadius + applySupportBoundaryTaper :1038-1058, :957-982
//                           -> crop_sum_kernel, combine_kernel
//   estimateFirstMinimumRadius :865-955 -> profile_kernel + first_zero_scan_kernel
//
// All wavelengths of a bank run in the same launches (blockIdx.y / .z is the
// wavelength).  No stage returns to the host.  The canvas of a wavelength is
// overwritten stage by stage: resampled value -> shaped value (shape_stats) ->
// shaped * taper inside the crop box, 0 outside (crop_sum); the final,
// normalised kernel is that value / (s3 * s4).
#include <algorithm>
#include <climits>

#include "ld_internal.h"
#include "ld_launch.cuh"

namespace ld {
namespace {

constexpr int kTile = 32;       // canvas tile side for the per-pixel kernels
constexpr int kRingSpan = 64;   // ring indices one 32x32 tile can touch
// The ring-statistics passes (resample, shape_stats) take 32 x 128 tiles:
// sixteen rows per thread amortise each CTA's ring setup, flush and sums.
constexpr int kTallH = 128;
constexpr int kRingSpanTall = 160;  // >= sqrt(31^2 + 127^2) + 3

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block-wide sum of one double; result valid in thread 0.
__device__ double block_sum(double v) {
    __shared__ double part[32];
    const int tid = threadIdx.x + threadIdx.y * blockDim.x;
    const int lane = tid & 31, warp = tid >> 5;
    v = warp_sum(v);
    const int nwarps = (blockDim.x * blockDim.y + 31) >> 5;
    __syncthreads();
    if (lane == 0) part[warp] = v;
    __syncthreads();
    double r = 0.0;
    if (warp == 0) {
        r = lane < nwarps ? part[lane] : 0.0;
        r = warp_sum(r);
    }
    return r;
}

// Inclusive segmented scan over the runs of equal slots in consecutive lanes:
// leaves each run's sum (and maximum) in v (and m) of its last lane, for
// which it returns true.  `far`: lanes whose `o` lanes before them belong to
// their run, i.e. the step of distance o has work; off the canvas's axes a
// run is one to three pixels long, so most rows need one or two steps.
template <bool PEAK>
__device__ __forceinline__ bool warp_runs_scan(int slot, float& v, float& m) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int prev = __shfl_up_sync(full, slot, 1);
    const unsigned heads = __ballot_sync(full, lane == 0 || prev != slot);
    unsigned far = ~heads;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        if (far == 0u) break;  // uniform
        const float t = __shfl_up_sync(full, v, o);
        const float u = PEAK ? __shfl_up_sync(full, m, o) : 0.0f;
        if ((far >> lane) & 1u) {
            v += t;
            if (PEAK) m = fmaxf(m, u);
        }
        far &= far << o;
    }
    return lane == 31 || ((heads >> (lane + 1)) & 1u) != 0u;
}

// Adds each lane's v to ring[slot] (and, with PEAK, maxes its top into
// peak[slot] as float bits) where the lanes' slots form runs of equal values
// in consecutive lanes (slot < 0: nothing to add), v >= 0.  A warp is 32
// pixels of a canvas row, along which the ring index is monotonic on each
// side of the centre, so equal slots are contiguous.  One inclusive
// segmented scan over the warp (warp_runs_scan) gives each run's sum (and
// maximum) in its last lane, which adds it with one shared-memory atomic.
template <bool PEAK>
__device__ __forceinline__ void warp_runs_accumulate(int slot, float v, float top, float* ring, unsigned int* peak) {
    if (warp_runs_scan<PEAK>(slot, v, top) && slot >= 0) {
        if (v != 0.0f) atomicAdd(&ring[slot], v);
        if (PEAK && top != 0.0f) atomicMax(&peak[slot], __float_as_uint(top));
    }
}

// ---- pupil, once per bank --------------------------------------------------------
__global__ void __launch_bounds__(256) pupil_pre_kernel(PsfBankArgs a) {
    stream_order();
    const int n = a.pupil.size;
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n * n) return;
    const int x = i % n, y = i / n;
    const float amp = pupil_amplitude(a.pupil, x, y);
    float phi0 = 0.0f, z4 = 0.0f, valid = 0.0f;
    if (amp > 0.0f) pupil_phase_split(a.pupil, a.base_phase, x, y, &phi0, &z4, &valid);
    a.pupil_pre[i] = make_float4(amp, phi0, z4, valid);
}

// ---- raw PSF: row pass ---------------------------------------------------------
// grid (row_n, B).  Pupil row y = row_lo + blockIdx.x, embedded at (S-N_p)/2 of
// a length-S row; the field A exp(i 2 pi phi) is generated in the fill, the
// window columns are written by the drain.
template <int E>
__global__ void __launch_bounds__(E >= kE25 ? kE25MaxThreads : kE16MaxThreads, 1) psf_rows_kernel(PsfBankArgs a) {
    stream_order();
    extern __shared__ float2 smem[];
    const int yr = blockIdx.x;
    const int y = a.row_lo + yr;
    const int b = blockIdx.y;
    const WavelengthInfo* w = a.wl + b;
    const int np = a.pupil.size;
    const int off = a.off;
    const int enabled = w->phase.enabled;
    const float c4 = w->phase.c[4];
    const float4* pre = a.pupil_pre + static_cast<size_t>(y) * np;
    smem_fill<1>(smem, a.S, [=](int idx, int) -> float2 {
        const int x = idx - off;
        if (x < 0 || x >= np) return make_float2(0.0f, 0.0f);
        const float4 q = pre[x];
        if (q.x <= 0.0f) return make_float2(0.0f, 0.0f);
        const float ph = (enabled && q.w != 0.0f) ? q.y + c4 * q.z : 0.0f;
        if (ph == 0.0f) return make_float2(q.x, 0.0f);
        float sn, cs;
        sincosf(ph * 2.0f * kPiF, &sn, &cs);
        return make_float2(q.x * cs, q.x * sn);
    });
    fft_run<E, 1, false>(a.plan_s, smem);
    const int wn = w->win_n;
    const int wx0 = w->win_x0;
    const int S = a.S;
    float2* out = a.rows + (static_cast<size_t>(b) * a.row_n + yr) * a.win_stride;
    for (int wx = threadIdx.x; wx < wn; wx += blockDim.x) {
        int u = wx0 + wx + a.half;  // shifted column X -> unshifted (X + S/2) mod S
        if (u >= S) u -= S;
        out[wx] = smem[u];
    }
}

// ---- raw PSF: column pass + |.|^2 + fftshift window -----------------------------
// grid (ceil(win/C), B).  Columns X0..X0+C of the window; only the pupil rows
// that can be non-zero are read, |F|^2 of the window rows is written.
template <int E, int C>
__global__ void __launch_bounds__(E >= kE25 ? kE25MaxThreads : kE16MaxThreads, 1) psf_cols_kernel(PsfBankArgs a) {
    stream_order();
    extern __shared__ float2 smem[];
    const int b = blockIdx.y;
    const WavelengthInfo* w = a.wl + b;
    const int wn = w->win_n;
    const int X0 = blockIdx.x * C;
    if (X0 >= wn) return;
    const int lo = a.off + a.row_lo;
    const int rn = a.row_n;
    const int stride = a.win_stride;
    const float2* in = a.rows + static_cast<size_t>(b) * rn * stride;
    float* outw = a.win + static_cast<size_t>(b) * stride * stride;
    smem_fill<C>(smem, a.S, [=](int idx, int col) -> float2 {
        const int g = idx - lo;
        const int X = X0 + col;
        if (g < 0 || g >= rn || X >= wn) return make_float2(0.0f, 0.0f);
        return in[static_cast<size_t>(g) * stride + X];
    });
    fft_run<E, C, false>(a.plan_s, smem);
    const int S = a.S;
    const int wy0 = w->win_x0;
    double esum = 0.0;
    for (int i = threadIdx.x; i < wn * C; i += blockDim.x) {
        const int wy = i / C, col = i % C;
        const int X = X0 + col;
        if (X >= wn) continue;
        int v = wy0 + wy + a.half;  // shifted row Y -> unshifted (Y + S/2) mod S
        if (v >= S) v -= S;
        const float2 f = smem[v * C + col];
        const float I = f.x * f.x + f.y * f.y;
        outw[static_cast<size_t>(wy) * stride + X] = I;
        esum += I;
    }
    if (a.want_energy) {
        const double tot = block_sum(esum);
        if (threadIdx.x == 0) atomicAdd(&a.scalars[b].energy, tot);
    }
}

// ---- lambda-rescale -----------------------------------------------------------------
struct Window {
    const float* p;
    int stride, x0, n, S;
};

// First ring index a 32 x th tile can touch, for a centre at (c, c) and ring
// indices clamped to `cap`: every pixel of the tile has a ring index in
// [base, base + span) with span <= the tile's diagonal + 3 (kRingSpan for
// 32 x 32 tiles, kRingSpanTall for the 32 x 128 tiles of the ring-statistics
// passes).
__device__ __forceinline__ int tile_ring_base(int tx0, int ty0, int c, int cap, int th = kTile) {
    const int dx = tx0 > c ? tx0 - c : (tx0 + kTile - 1 < c ? c - (tx0 + kTile - 1) : 0);
    const int dy = ty0 > c ? ty0 - c : (ty0 + th - 1 < c ? c - (ty0 + th - 1) : 0);
    const float r = sqrtf(static_cast<float>(dx * dx + dy * dy));
    return min(cap, max(0, static_cast<int>(r) - 1));
}

// The column half of a bilinear sample of the |F|^2 window at x
// (sampleSquareBilinear, LensDiffCpuReference.cpp:316-336; the window covers
// every pixel the kernel touches): the same for every row a thread samples.
struct ColTap {
    bool in;       // x inside [0, S - 1]
    int ax0, ax1;  // window columns of x0 and x1
    float tx;
};
__device__ __forceinline__ ColTap col_tap(const Window& w, float x) {
    ColTap c;
    c.in = !(x < 0.0f || x > static_cast<float>(w.S - 1));
    const int x0 = static_cast<int>(floorf(x));
    const int x1 = min(x0 + 1, w.S - 1);
    c.tx = x - static_cast<float>(x0);
    const int hi = w.n - 1;
    c.ax0 = min(max(x0 - w.x0, 0), hi);
    c.ax1 = min(max(x1 - w.x0, 0), hi);
    return c;
}
// FUSED (anisotropy gain 1): reshapeAnisotropy (LensDiffCpuReference.cpp:1122-1134)
// then gives mean + (base - mean) * 1, the base kernel itself up to one
// rounding, so the canvas keeps the resampled values unnormalised and the
// rescale takes the shaped kernel's statistics that shape_stats_kernel takes
// otherwise (s3 = s1, the ceil(r) ring energies and peaks, the peak) in
// place of the round(r) ring sums, which only the Split look's ring means
// need (ring_sums_kernel, run when a Split render first uses the bank).

// Ring statistics of one λ-rescale tile, and its staged window pixels.
template <bool FUSED>
struct RingSmem {
    float ring[kRingSpanTall];  // FUSED: the ceil(r) ring energies, else the round(r) sums
    unsigned int ring_p[FUSED ? kRingSpanTall : 1];
    __device__ void clear(int tid) {
        for (int i = tid; i < kRingSpanTall; i += 256) {
            ring[i] = 0.0f;
            if constexpr (FUSED) ring_p[i] = 0u;
        }
    }
};

// Ring slot of canvas pixel (x, y) relative to the tile's first ring `rbase`
// (-1: no pixel): ceil(r) (FUSED) or round(r) of its distance to the centre.
template <bool FUSED>
__device__ __forceinline__ int ring_slot(bool in, float dx, float dy, int R, int rbase) {
    if (!in) return -1;
    const float rr = sqrtf(dx * dx + dy * dy);
    return min(R, static_cast<int>(FUSED ? ceilf(rr) : roundf(rr))) - rbase;
}

// The peak and the sum of a tile's pixels go to the wavelength's statistics.
template <bool FUSED>
__device__ __forceinline__ void resample_totals(const PsfBankArgs& a, int b, float lsum, unsigned int lpeak, int tid) {
    if constexpr (FUSED) {
        for (int o = 16; o > 0; o >>= 1) lpeak = max(lpeak, __shfl_xor_sync(0xffffffffu, lpeak, o));
        if ((tid & 31) == 0 && lpeak != 0u) atomicMax(&a.scalars[b].peak, lpeak);
    }
    const double tot = block_sum(static_cast<double>(lsum));
    if (tid == 0) {
        atomicAdd(&a.scalars[b].s1, tot);
        if constexpr (FUSED) atomicAdd(&a.scalars[b].s3, tot);
    }
}

// The end of one wavelength's tile: the CTA's ring sums and peaks, the peak
// and the canvas sum go to the wavelength's global statistics.
template <bool FUSED>
__device__ __forceinline__ void resample_flush(const PsfBankArgs& a, int b, int rbase, RingSmem<FUSED>& sm,
                                               float lsum, unsigned int lpeak, int tid) {
    __syncthreads();
    const int R = a.R;
    const size_t ro = static_cast<size_t>(b) * (R + 1);
    for (int i = tid; i < kRingSpanTall; i += 256) {
        if (rbase + i > R) continue;
        if (sm.ring[i] != 0.0f)
            atomicAdd(&(FUSED ? a.ring_ceil : a.ring_round)[ro + rbase + i], static_cast<double>(sm.ring[i]));
        if constexpr (FUSED) {
            if (sm.ring_p[i] != 0u) atomicMax(&a.ring_peak[ro + rbase + i], sm.ring_p[i]);
        }
    }
    resample_totals<FUSED>(a, b, lsum, lpeak, tid);
}

// ---- lambda-rescale without a box filter ----------------------------------------
// The canvas samples the |F|^2 window at most one window pixel apart
// (scaleFactor >= 1).  A CTA takes a 32 x th tile of the canvas's quadrant
// dx, dy >= 0 together with its three mirror images: the four pixels
// (+-dx, +-dy) lie on one ring, so the ring slot and the segmented scan of the
// ring statistics run once for the four.  The window pixels under the four
// images are staged in shared memory.  A warp walks th / 8 consecutive canvas
// rows; the rows' sample positions are uniform in the warp, so the two
// horizontally interpolated window rows a sample blends are kept in registers
// until the position moves to the next window row (every 1 / inv_scale
// canvas rows).  Bound by instruction issue (80 M warp instructions, 68 % of
// the issue slots): 113 us for 31 wavelengths at K = 1025 (168 us for tiles
// without the mirror images, two wavelengths at a time, every sample from
// four shared-memory reads).
constexpr int kQuadH = 128;

// Window indices [lo, hi] that canvas offsets d0 .. d1 (d0 <= d1) from the
// centre sample, one more on each side so that the span holds whatever the
// rounding of the sample positions.
__device__ __forceinline__ void quad_span(const Window& w, float rc, float inv, float d0, float d1, int* lo, int* hi) {
    const float p0 = rc + d0 * inv, p1 = rc + d1 * inv;
    const int whi = w.n - 1;
    const int a0 = static_cast<int>(floorf(fmaxf(p0, 0.0f)));
    const int a1 = min(static_cast<int>(floorf(fminf(fmaxf(p1, 0.0f), static_cast<float>(w.S - 1)))) + 1, w.S - 1);
    *lo = min(max(a0 - 1 - w.x0, 0), whi);
    *hi = min(max(a1 + 1 - w.x0, 0), whi);
}

// Staged pixels per box side for `n` canvas pixels sampled `inv` apart
// (quad_span's count, with one for rounding).
__host__ __device__ constexpr int quad_stage(int n, float inv) { return static_cast<int>((n - 1) * inv) + 7; }

// Tile (tx, ty) of wavelength b; block (32, 8).  Shared memory: the warps' ring
// statistics, then the staged boxes [row image][column image][sh][sw].
// Along a quadrant's row the ring index only grows, so a row's runs have
// distinct slots: each warp adds them to ring statistics of its own with
// plain loads and stores.
constexpr int kRingSpanQuad = 136;  // >= sqrt(31^2 + 127^2) + 3
constexpr size_t kQuadRingBytes = 8 * kRingSpanQuad * sizeof(float2);

template <bool FUSED>
__device__ __forceinline__ void resample_quad(const PsfBankArgs& a, int tx, int ty, int b, int th, int sw, int sh,
                                              float2* smem) {
    float2(*ring)[kRingSpanQuad] = reinterpret_cast<float2(*)[kRingSpanQuad]>(smem);  // per warp: sums and peaks
    float* stage = reinterpret_cast<float*>(smem + 8 * kRingSpanQuad);
    const WavelengthInfo* wi = a.wl + b;
    const int lane = threadIdx.x;
    const int tid = lane + threadIdx.y * 32;
    const int K = a.K, R = a.R;
    const int tx0 = tx * kTile, ty0 = ty * th;  // offsets from the centre
    const int rbase = tile_ring_base(tx0, ty0, 0, R, th);
    float2* wring = ring[threadIdx.y];
    for (int i = lane; i < kRingSpanQuad; i += 32) wring[i] = make_float2(0.0f, 0.0f);
    const Window w{a.win + static_cast<size_t>(b) * a.win_stride * a.win_stride, a.win_stride, wi->win_x0,
                   wi->win_n, a.S};
    const float inv = wi->inv_scale;
    const float rc = a.raw_center;
    // [0]: the images at +dx / +dy, [1]: at -dx / -dy
    int cx[2], cy[2], hx[2], hy[2];
    const float fx0 = static_cast<float>(tx0), fx1 = static_cast<float>(min(tx0 + kTile - 1, R));
    const float fy0 = static_cast<float>(ty0), fy1 = static_cast<float>(min(ty0 + th - 1, R));
    quad_span(w, rc, inv, fx0, fx1, &cx[0], &hx[0]);
    quad_span(w, rc, inv, -fx1, -fx0, &cx[1], &hx[1]);
    quad_span(w, rc, inv, fy0, fy1, &cy[0], &hy[0]);
    quad_span(w, rc, inv, -fy1, -fy0, &cy[1], &hy[1]);
#pragma unroll
    for (int v = 0; v < 2; ++v) {
        const int bh = min(hy[v] - cy[v] + 1, sh);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int bw = min(hx[h] - cx[h] + 1, sw);
            float* st = stage + (v * 2 + h) * sh * sw;
            const float* src = w.p + static_cast<size_t>(cy[v]) * w.stride + cx[h];
            for (int r = threadIdx.y; r < bh; r += 8)
                for (int c = lane; c < bw; c += 32) st[r * sw + c] = __ldg(src + r * w.stride + c);
        }
    }
    __syncthreads();
    const int ix = tx0 + lane;
    const bool in = ix <= R;
    const bool mirror = in && ix > 0;  // column 0 has no mirror image
    const float dx = static_cast<float>(ix);
    const ColTap ct[2] = {col_tap(w, rc + dx * inv), col_tap(w, rc - dx * inv)};
    int s0[2], s1[2];  // the taps' columns in the staged boxes
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        s0[h] = min(max(ct[h].ax0 - cx[h], 0), sw - 1) + h * sh * sw;
        s1[h] = min(max(ct[h].ax1 - cx[h], 0), sw - 1) + h * sh * sw;
    }
    const bool use[2] = {in && ct[0].in, mirror && ct[1].in};
    // the two window rows under a canvas row, interpolated at the thread's two
    // columns (h0, h1 [row image][column image]), and the window row (as a
    // float) they belong to
    float h0[2][2] = {}, h1[2][2] = {}, at[2] = {-1.0f, -1.0f};
    const float lim = static_cast<float>(w.S - 1);
    const int rows = th / 8;
    const int iy0 = ty0 + threadIdx.y * rows;
    float* const canvas = a.canvas + static_cast<size_t>(b) * K * K + static_cast<size_t>(R) * K + R;
    float* up = canvas + static_cast<ptrdiff_t>(iy0) * K;   // row +dy, at the centre column
    float* down = canvas - static_cast<ptrdiff_t>(iy0) * K; // row -dy
    // ceil(sqrtf(n)) of integers n < 2^24 is exact, so the slot follows n by
    // comparison with the squares; else (and for round(r)) by the square root
    const bool exact = FUSED && R < 2048;
    int n = ix * ix + iy0 * iy0;
    int ring_i = exact ? static_cast<int>(ceilf(sqrtf(static_cast<float>(n)))) : 0;
    float lsum = 0.0f;  // this thread's pixels; one double add per thread at the flush
    float lpeak = 0.0f;
    for (int i = 0; i < rows; ++i) {
        const int iy = iy0 + i;
        if (iy > R) break;  // uniform: a warp walks canvas rows
        const float dy = static_cast<float>(iy);
        float sum = 0.0f, m = 0.0f;
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            if (v == 1 && iy == 0) break;  // row 0 has no mirror image
            const float yy = v == 0 ? rc + dy * inv : rc - dy * inv;
            const bool ok = !(yy < 0.0f || yy > lim);
            const float fl = floorf(yy);
            const float f = yy - fl;
            if (ok && fl != at[v]) {  // uniform
                const int y0 = static_cast<int>(fl);
                const int hi = w.n - 1;
                const int o = v * 2 * sh;
                const int r0 = (min(min(max(y0 - w.x0, 0), hi) - cy[v], sh - 1) + o) * sw;
                const int r1 = (min(min(max(min(y0 + 1, w.S - 1) - w.x0, 0), hi) - cy[v], sh - 1) + o) * sw;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float v00 = stage[r0 + s0[h]], v10 = stage[r0 + s1[h]];
                    const float v01 = stage[r1 + s0[h]], v11 = stage[r1 + s1[h]];
                    h0[v][h] = v00 + (v10 - v00) * ct[h].tx;
                    h1[v][h] = v01 + (v11 - v01) * ct[h].tx;
                }
                at[v] = fl;
            }
            float* row = v == 0 ? up : down;
            const float v0 = ok && use[0] ? h0[v][0] + (h1[v][0] - h0[v][0]) * f : 0.0f;
            const float v1 = ok && use[1] ? h0[v][1] + (h1[v][1] - h0[v][1]) * f : 0.0f;
            if (in) row[ix] = v0;
            if (mirror) row[-ix] = v1;
            sum += v0 + v1;
            m = fmaxf(m, fmaxf(v0, v1));
        }
        up += K;
        down -= K;
        lsum += sum;
        lpeak = fmaxf(lpeak, m);
        int slot = -1;
        if (exact) {
            if (in) slot = min(R, ring_i) - rbase;
            n += 2 * iy + 1;  // the next row's
            ring_i += n > ring_i * ring_i ? 1 : 0;
        } else {
            slot = ring_slot<FUSED>(in, dx, dy, R, rbase);
        }
        if (warp_runs_scan<FUSED>(slot, sum, m) && slot >= 0) {
            float2 e = wring[slot];
            e.x += sum;
            if constexpr (FUSED) e.y = fmaxf(e.y, m);
            wring[slot] = e;
        }
        __syncwarp();
    }
    __syncthreads();
    const size_t ro = static_cast<size_t>(b) * (R + 1);
    for (int i = tid; i < kRingSpanQuad; i += 256) {
        if (rbase + i > R) continue;
        float e = 0.0f, p = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            e += ring[k][i].x;
            p = fmaxf(p, ring[k][i].y);
        }
        if (e != 0.0f) atomicAdd(&(FUSED ? a.ring_ceil : a.ring_round)[ro + rbase + i], static_cast<double>(e));
        if (FUSED && p != 0.0f) atomicMax(&a.ring_peak[ro + rbase + i], __float_as_uint(p));
    }
    resample_totals<FUSED>(a, b, lsum, __float_as_uint(lpeak), tid);
}

// ---- box-filtered lambda-rescale ------------------------------------------------
// Samples more than one window pixel apart (scaleFactor < 1) are the mean of
// taps x taps bilinear samples (sampleSquareFiltered,
// LensDiffCpuReference.cpp:338-353).  The mean is separable: along each axis
// the taps' bilinear weights add up to weights on a run of at most
// kFilterSpan window pixels (taps <= 6, footprint <= 20: five steps of at
// most 20 / 6 and the two pixels of a tap).  A CTA forms the column weights
// of its 32 canvas columns and the row weights of its th canvas rows once;
// each warp then takes a canvas row at a time: the run of window rows into
// one weighted row (coalesced: lanes are window columns), from which its 32
// lanes take their weighted runs.  Per canvas pixel about footprint x run
// multiply-adds instead of taps^2 bilinear samples of ~40 instructions.
// Bound by the latency of the window reads: 71 us for 16 wavelengths at
// K = 513 with footprints 3.3-5.7 and PSF size 1024 (186 us sampling tap by
// tap), 20 us for 3 at K = 257 with footprints 5.2-9.1 (77 us).
constexpr int kFilterSpan = 20;
constexpr int kFilterRow = 672;  // >= 31 * 20 + 17 + 3 window columns under 32 canvas columns

struct FilterSmem {
    float row[8][kFilterRow];          // per warp: the window rows of one canvas row, weighted
    float cw[kFilterSpan][kTile];      // column weights [run][canvas column]
    float rw[kTallH][kFilterSpan];     // row weights [canvas row][run]
    int r0[kTallH], rn[kTallH];        // first window row of a canvas row's run, and its length
    int cx0, span;                     // window columns the tile reads
    float ring[2 * kRingSpanTall];     // RingSmem
};

// Weights of the taps around coordinate p on a run of window pixels from
// *first on (w[j * stride], j < the returned length; 0: no tap inside
// [0, S - 1], where sampleSquareBilinear is zero).
__device__ __forceinline__ int tap_weights(const Window& win, float p, float footprint, int taps, float step, float* w,
                                           int stride, int* first) {
    for (int j = 0; j < kFilterSpan; ++j) w[j * stride] = 0.0f;
    const float lim = static_cast<float>(win.S - 1);
    const int hi = win.n - 1;
    int lo = 0, n = 0;
    for (int t = 0; t < taps; ++t) {
        const float q = p + ((static_cast<float>(t) + 0.5f) * step - footprint * 0.5f);
        if (q < 0.0f || q > lim) continue;
        const int i0 = static_cast<int>(floorf(q));
        const float f = q - static_cast<float>(i0);
        const int a0 = min(max(i0 - win.x0, 0), hi);
        const int a1 = min(max(min(i0 + 1, win.S - 1) - win.x0, 0), hi);
        if (n == 0) lo = a0;
        const int j0 = min(a0 - lo, kFilterSpan - 1), j1 = min(a1 - lo, kFilterSpan - 1);
        w[j0 * stride] += 1.0f - f;
        w[j1 * stride] += f;
        n = j1 + 1;
    }
    *first = lo;
    return n;
}

// The 32 x th canvas tile (tx, ty) of wavelength b; block (32, 8).
template <bool FUSED>
__device__ __forceinline__ void resample_filtered(const PsfBankArgs& a, int tx, int ty, int b, int th,
                                                  FilterSmem& fs) {
    RingSmem<FUSED>& sm = *reinterpret_cast<RingSmem<FUSED>*>(fs.ring);
    const WavelengthInfo* wi = a.wl + b;
    const int tid = threadIdx.x + threadIdx.y * 32;
    const int K = a.K, R = a.R;
    const int tx0 = tx * kTile, ty0 = ty * th;
    const int rbase = tile_ring_base(tx0, ty0, R, R, th);
    sm.clear(tid);
    const Window w{a.win + static_cast<size_t>(b) * a.win_stride * a.win_stride, a.win_stride, wi->win_x0,
                   wi->win_n, a.S};
    const float kc = static_cast<float>(K - 1) * 0.5f;
    const float inv = wi->inv_scale;
    const int taps = wi->taps;
    const float step = wi->step;
    const float rc = a.raw_center;
    const int lane = threadIdx.x;
    const int x = tx0 + lane;
    const bool in = x < K;
    const float dx = static_cast<float>(x) - kc;
    int c0 = 0, cn = 0;
    if (threadIdx.y == 7) {  // the last warp: column weights (the rows' threads come first)
        if (in) cn = tap_weights(w, rc + dx * inv, inv, taps, step, &fs.cw[0][lane], kTile, &c0);
        const int lo = __reduce_min_sync(0xffffffffu, cn > 0 ? c0 : INT_MAX);
        const int hi = __reduce_max_sync(0xffffffffu, cn > 0 ? c0 + cn : 0);
        if (lane == 0) {
            fs.cx0 = hi > 0 ? lo : 0;
            fs.span = hi > 0 ? min(hi - lo, kFilterRow) : 0;
        }
        fs.row[0][lane] = __int_as_float(c0);  // handed to the other warps, which share the columns
        fs.row[1][lane] = __int_as_float(cn);
    }
    for (int r = tid; r < th; r += 224) {
        if (tid >= 224) break;
        const float dy = static_cast<float>(ty0 + r) - kc;
        fs.rn[r] = ty0 + r < K ? tap_weights(w, rc + dy * inv, inv, taps, step, fs.rw[r], 1, &fs.r0[r]) : 0;
    }
    __syncthreads();
    const int cx0 = fs.cx0, span = fs.span;
    c0 = __float_as_int(fs.row[0][lane]) - cx0;
    cn = __float_as_int(fs.row[1][lane]);
    const int cmax = __reduce_max_sync(0xffffffffu, cn);
    __syncthreads();  // row[] is free
    const float area = static_cast<float>(taps * taps);
    float* canvas = a.canvas + static_cast<size_t>(b) * K * K;
    float* vrow = fs.row[threadIdx.y];
    float lsum = 0.0f;
    unsigned int lpeak = 0u;
    const int rows = th / 8;
    for (int i = 0; i < rows; ++i) {
        const int r = threadIdx.y + 8 * i;
        const int y = ty0 + r;
        if (y >= K) break;  // uniform: a warp is one canvas row
        const int rn = fs.rn[r];
        float v = 0.0f;
        if (rn > 0 && span > 0) {  // uniform
            const float* base = w.p + static_cast<size_t>(fs.r0[r]) * w.stride + cx0;
            // kU window columns per lane, kJ rows at a time: twenty reads in
            // flight per lane, since the windows come from L2 or HBM (with
            // eight in flight the HD bank took 103 us instead of 69)
            constexpr int kU = 2, kJ = 10;
            for (int c = lane; c < span; c += 32 * kU) {
                const int o0 = c, o1 = min(c + 32, span - 1);
                float acc0 = 0.0f, acc1 = 0.0f;
                for (int j0 = 0; j0 < rn; j0 += kJ) {
                    float v0[kJ], v1[kJ];
#pragma unroll
                    for (int j = 0; j < kJ; ++j) {
                        const float* p = base + min(j0 + j, rn - 1) * w.stride;  // past the run: weight 0
                        v0[j] = __ldg(p + o0);
                        v1[j] = __ldg(p + o1);
                    }
#pragma unroll
                    for (int j = 0; j < kJ; ++j) {
                        acc0 += fs.rw[r][j0 + j] * v0[j];
                        acc1 += fs.rw[r][j0 + j] * v1[j];
                    }
                }
                vrow[c] = acc0;
                if (c + 32 < span) vrow[c + 32] = acc1;
            }
            __syncwarp();
            float sum = 0.0f;
            for (int j = 0; j < cmax; ++j)
                if (j < cn) sum += fs.cw[j][lane] * vrow[c0 + j];
            v = sum / area;
            __syncwarp();
        }
        if (in) canvas[static_cast<size_t>(y) * K + x] = v;
        lsum += v;
        if constexpr (FUSED) lpeak = max(lpeak, __float_as_uint(v));
        const float dy = static_cast<float>(y) - kc;
        warp_runs_accumulate<FUSED>(ring_slot<FUSED>(in, dx, dy, R, rbase), v, v, sm.ring, sm.ring_p);
    }
    resample_flush<FUSED>(a, b, rbase, sm, lsum, lpeak, tid);
}

// The rescale of a whole bank, 1-D grid, block (32, 8): nq quadrant tiles
// (qx x qy per wavelength), then the box-filtered tiles (fx x fy per
// wavelength).  Each wavelength's work is in the tiles of its own kind.
struct ResampleGrid {
    int nq, qx, qy, qth, sw, sh;
    int fx, fy, fth;
};
template <bool FUSED>
__global__ void __launch_bounds__(256) resample_kernel(PsfBankArgs a, ResampleGrid g) {
    stream_order();
    extern __shared__ float2 smem[];
    int i = blockIdx.x;
    if (i < g.nq) {
        const int b = i / (g.qx * g.qy);
        if (a.wl[b].taps != 0) return;
        i -= b * g.qx * g.qy;
        resample_quad<FUSED>(a, i % g.qx, i / g.qx, b, g.qth, g.sw, g.sh, smem);
    } else {
        i -= g.nq;
        const int b = i / (g.fx * g.fy);
        if (a.wl[b].taps == 0) return;
        i -= b * g.fx * g.fy;
        resample_filtered<FUSED>(a, i % g.fx, i / g.fx, b, g.fth, *reinterpret_cast<FilterSmem*>(smem));
    }
}

// ---- lambda-rescale of the FP16 form's banks with a box filter ------------------
// The FP16 form rounds its kernel spectra to half, where a canvas that differs
// in FP32's last bits moves stored values to their neighbours: with
// resample_filtered's separable weights in place of the tap-by-tap mean, and
// the statistics that scale the kernel summed in another order, a small
// log-encoded frame moved by 7e-5 of its norm, at the same error against FP64.
// A bank with a box filter is therefore sampled tap by tap, and summed, over
// 32 x 128 tiles, one wavelength a tile: 125 us for 16 wavelengths at K = 513
// with footprints 3.3-5.7 (76 us separably, 193 us with the columns of a tap
// formed anew for every sample).  (In a bank without a box filter
// resample_quad's tiles take the same samples, and their sums move the outputs
// by up to 1.7e-5, most by under 5e-6.)

// The columns of a pixel's taps (the x terms of sampleSquareBilinear,
// LensDiffCpuReference.cpp:316-336): the same for every row a thread samples.
constexpr int kTaps = 6;
__device__ __forceinline__ void tap_columns(const Window& w, float px, float footprint, float step, ColTap (&ct)[kTaps]) {
#pragma unroll
    for (int t = 0; t < kTaps; ++t) ct[t] = col_tap(w, px + ((static_cast<float>(t) + 0.5f) * step - footprint * 0.5f));
}

// The mean of taps x taps bilinear samples (sampleSquareFiltered,
// LensDiffCpuReference.cpp:338-353), a row of taps at a time; a tap outside
// [0, S - 1] adds zero.
__device__ __forceinline__ float sample_taps(const Window& w, const ColTap (&ct)[kTaps], float py, float footprint,
                                             int taps, float step) {
    const float lim = static_cast<float>(w.S - 1);
    const int hi = w.n - 1;
    float sum = 0.0f;
    for (int t = 0; t < taps; ++t) {  // uniform: a warp is one canvas row
        const float y = py + ((static_cast<float>(t) + 0.5f) * step - footprint * 0.5f);
        if (y < 0.0f || y > lim) continue;
        const int y0 = static_cast<int>(floorf(y));
        const float ty = y - static_cast<float>(y0);
        const float* r0 = w.p + static_cast<size_t>(min(max(y0 - w.x0, 0), hi)) * w.stride;
        const float* r1 = w.p + static_cast<size_t>(min(max(min(y0 + 1, w.S - 1) - w.x0, 0), hi)) * w.stride;
#pragma unroll
        for (int u = 0; u < kTaps; ++u) {
            if (u >= taps || !ct[u].in) continue;
            const float v00 = __ldg(r0 + ct[u].ax0), v10 = __ldg(r0 + ct[u].ax1);
            const float v01 = __ldg(r1 + ct[u].ax0), v11 = __ldg(r1 + ct[u].ax1);
            const float vx0 = v00 + (v10 - v00) * ct[u].tx;
            const float vx1 = v01 + (v11 - v01) * ct[u].tx;
            sum += vx0 + (vx1 - vx0) * ty;
        }
    }
    return sum / static_cast<float>(taps * taps);
}

// One bilinear sample with the column half precomputed (identical arithmetic).
__device__ __forceinline__ float sample_row(const Window& w, const ColTap& c, float y) {
    if (!c.in || y < 0.0f || y > static_cast<float>(w.S - 1)) return 0.0f;
    const int y0 = static_cast<int>(floorf(y));
    const int y1 = min(y0 + 1, w.S - 1);
    const float ty = y - static_cast<float>(y0);
    const int hi = w.n - 1;
    const float* r0 = w.p + min(max(y0 - w.x0, 0), hi) * w.stride;
    const float* r1 = w.p + min(max(y1 - w.x0, 0), hi) * w.stride;
    const float v00 = __ldg(r0 + c.ax0), v10 = __ldg(r0 + c.ax1);
    const float v01 = __ldg(r1 + c.ax0), v11 = __ldg(r1 + c.ax1);
    const float vx0 = v00 + (v10 - v00) * c.tx;
    const float vx1 = v01 + (v11 - v01) * c.tx;
    return vx0 + (vx1 - vx0) * ty;
}

// Window pixels staged per tile of unfiltered samples (at most one window pixel
// apart), one more on each side so that the span holds whatever the rounding
// of the sample positions.
constexpr int kStageW = kTile + 4, kStageH = kTallH + 4;

// Rows / columns of the window that canvas coordinates c0 .. c1 sample
// (x0 .. x1 of the first and last sample, clamped to the
// window as it clamps them): [lo, hi] in window indices.
__device__ __forceinline__ void stage_span(const Window& w, float rc, float kc, float inv, int c0, int c1, int* lo,
                                           int* hi) {
    const float p0 = rc + (static_cast<float>(c0) - kc) * inv;
    const float p1 = rc + (static_cast<float>(c1) - kc) * inv;
    const int whi = w.n - 1;
    const int a0 = static_cast<int>(floorf(fmaxf(p0, 0.0f)));
    const int a1 = min(static_cast<int>(floorf(fminf(fmaxf(p1, 0.0f), static_cast<float>(w.S - 1)))) + 1, w.S - 1);
    *lo = min(max(a0 - 1 - w.x0, 0), whi);
    *hi = min(max(a1 + 1 - w.x0, 0), whi);
}

// Statistics of one tile, and the window pixels it samples.
template <bool FUSED>
struct TileSmem {
    RingSmem<FUSED> rings;
    float stage[kStageH][kStageW];
};

// The window pixels (rows cy0.., columns cx0..) a staged tile samples.
struct StageBox {
    int cx0, cy0, sw, sh;
};

// The staged box of wavelength `w`'s window for the tile at (tx0, ty0);
// ok = false when the samples are box-filtered or the span is too wide.
__device__ __forceinline__ bool stage_box(const Window& w, float rc, float kc, float inv, int taps, int tx0, int ty0,
                                          int K, StageBox* b) {
    if (taps != 0) return false;
    int cx1 = -1, cy1 = -1;
    stage_span(w, rc, kc, inv, tx0, min(tx0 + kTile, K) - 1, &b->cx0, &cx1);
    stage_span(w, rc, kc, inv, ty0, min(ty0 + kTallH, K) - 1, &b->cy0, &cy1);
    b->sw = cx1 - b->cx0 + 1;
    b->sh = cy1 - b->cy0 + 1;
    return b->sw <= kStageW && b->sh <= kStageH;
}

__device__ __forceinline__ void stage_load(const Window& w, const StageBox& b, float (*stage)[kStageW], int tid) {
    for (int i = tid; i < b.sw * b.sh; i += 256) {
        const int r = i / b.sw, c = i - r * b.sw;
        stage[r][c] = __ldg(w.p + static_cast<size_t>(b.cy0 + r) * w.stride + b.cx0 + c);
    }
}

// sample_row's arithmetic on staged pixels: the bilinear sample at window
// row coordinate yy of the column tap ct (sx0, sx1: its columns in the box).
__device__ __forceinline__ float staged_sample(const Window& w, const ColTap& ct, int sx0, int sx1, int cy0,
                                              const float (*stage)[kStageW], bool in, float yy) {
    const float lim = static_cast<float>(w.S - 1);
    if (!(in && ct.in && !(yy < 0.0f || yy > lim))) return 0.0f;
    const int hi = w.n - 1;
    const int y0 = static_cast<int>(floorf(yy));
    const int y1 = min(y0 + 1, w.S - 1);
    const float ty = yy - static_cast<float>(y0);
    const int sy0 = min(max(y0 - w.x0, 0), hi) - cy0;
    const int sy1 = min(max(y1 - w.x0, 0), hi) - cy0;
    const float v00 = stage[sy0][sx0], v10 = stage[sy0][sx1];
    const float v01 = stage[sy1][sx0], v11 = stage[sy1][sx1];
    const float vx0 = v00 + (v10 - v00) * ct.tx;
    const float vx1 = v01 + (v11 - v01) * ct.tx;
    return vx0 + (vx1 - vx0) * ty;
}

// One wavelength's 32 x 128 canvas tile; block (32, 8), 16 rows per thread.
// Unfiltered wavelengths of the bank stage the window pixels the tile reads in
// shared memory (stage_box); box-filtered samples, and any span too wide to
// stage, read the window directly.
template <bool FUSED>
__device__ void resample_tile(const PsfBankArgs& a, int b, int rbase, TileSmem<FUSED>& sm, int tid) {
    sm.rings.clear(tid);
    const WavelengthInfo* wi = a.wl + b;
    const int K = a.K, R = a.R;
    const int tx0 = blockIdx.x * kTile, ty0 = blockIdx.y * kTallH;
    const Window w{a.win + static_cast<size_t>(b) * a.win_stride * a.win_stride, a.win_stride, wi->win_x0,
                   wi->win_n, a.S};
    const float kc = static_cast<float>(K - 1) * 0.5f;
    const float inv = wi->inv_scale;
    const int taps = wi->taps;
    const float step = wi->step;
    const float rc = a.raw_center;
    float* canvas = a.canvas + static_cast<size_t>(b) * K * K;
    float lsum = 0.0f;  // this thread's pixels; one double add per thread at the flush
    unsigned int lpeak = 0u;
    const int x = tx0 + threadIdx.x;
    const bool in = x < K;
    const float dx = static_cast<float>(x) - kc;
    StageBox bx;
    if (stage_box(w, rc, kc, inv, taps, tx0, ty0, K, &bx)) {  // uniform per CTA
        stage_load(w, bx, sm.stage, tid);
        __syncthreads();
        const ColTap ct = col_tap(w, rc + dx * inv);
        const int sx0 = ct.ax0 - bx.cx0, sx1 = ct.ax1 - bx.cx0;
#pragma unroll 4
        for (int i = 0; i < kTallH / 8; ++i) {
            const int y = ty0 + threadIdx.y + 8 * i;
            if (y >= K) break;  // uniform: a warp is one canvas row
            const float dy = static_cast<float>(y) - kc;
            const float v = staged_sample(w, ct, sx0, sx1, bx.cy0, sm.stage, in, rc + dy * inv);
            if (in) canvas[static_cast<size_t>(y) * K + x] = v;
            lsum += v;
            if constexpr (FUSED) lpeak = max(lpeak, __float_as_uint(v));
            warp_runs_accumulate<FUSED>(ring_slot<FUSED>(in, dx, dy, R, rbase), v, v, sm.rings.ring, sm.rings.ring_p);
        }
    } else {
        __syncthreads();
        const ColTap ct = col_tap(w, rc + dx * inv);
        ColTap cts[kTaps];
        if (taps != 0) tap_columns(w, rc + dx * inv, inv, step, cts);
        for (int i = 0; i < kTallH / 8; ++i) {
            const int y = ty0 + threadIdx.y + 8 * i;
            if (y >= K) break;  // uniform: a warp is one canvas row (the last tile row is mostly past K)
            const float dy = static_cast<float>(y) - kc;
            float v = 0.0f;
            if (in) {
                v = taps == 0 ? sample_row(w, ct, rc + dy * inv) : sample_taps(w, cts, rc + dy * inv, inv, taps, step);
                canvas[static_cast<size_t>(y) * K + x] = v;
                lsum += v;
                if constexpr (FUSED) lpeak = max(lpeak, __float_as_uint(v));
            }
            warp_runs_accumulate<FUSED>(ring_slot<FUSED>(in, dx, dy, R, rbase), v, v, sm.rings.ring, sm.rings.ring_p);
        }
    }
    resample_flush<FUSED>(a, b, rbase, sm.rings, lsum, lpeak, tid);
}

// grid (ceil(K/32), ceil(K/128), B), block (32, 8): wavelength blockIdx.z.
template <bool FUSED>
__global__ void __launch_bounds__(256) resample_tile_kernel(PsfBankArgs a) {
    stream_order();
    __shared__ TileSmem<FUSED> sm;
    const int tid = threadIdx.x + threadIdx.y * 32;
    const int rbase = tile_ring_base(blockIdx.x * kTile, blockIdx.y * kTallH, a.R, a.R, kTallH);
    resample_tile<FUSED>(a, blockIdx.z, rbase, sm, tid);
}

// Sum over rings of the unnormalised azimuthal mean, i.e. the normaliser of
// azimuthalMeanKernel: sum_r count[r] * (ring[r] / s1) / count[r].
__device__ double mean_kernel_sum(const double* ring, const int* count, int R, double s1) {
    const int tid = threadIdx.x + threadIdx.y * blockDim.x;
    const int nth = blockDim.x * blockDim.y;
    double acc = 0.0;
    for (int r = tid; r <= R; r += nth) {
        const int c = max(1, count[r]);
        acc += static_cast<double>(count[r]) * ((ring[r] / s1) / c);
    }
    __shared__ double s2_shared;
    const double t = block_sum(acc);
    if (tid == 0) s2_shared = t;
    __syncthreads();
    return s2_shared;
}

// grid (B), block 256: s2 (the normaliser of azimuthalMeanKernel) and the
// normalised azimuthal mean of every round(r) ring, once per wavelength, for
// shape_stats_kernel to read.
__global__ void __launch_bounds__(256) ring_mean_kernel(PsfBankArgs a) {
    stream_order();
    const int b = blockIdx.x;
    const int R = a.R;
    const double s1 = a.scalars[b].s1;
    const double* rr = a.ring_round + static_cast<size_t>(b) * (R + 1);
    const double s2 = mean_kernel_sum(rr, a.count_round, R, s1);
    if (threadIdx.x == 0) a.scalars[b].s2 = s2;
    float* out = a.ring_mean + static_cast<size_t>(b) * (R + 1);
    for (int r = threadIdx.x; r <= R; r += blockDim.x)
        out[r] = static_cast<float>(((rr[r] / s1) / max(1, a.count_round[r])) / s2);
}

// grid (ceil(K/32), ceil(K/128), B), block (32, 8): the round(r) ring sums
// of a canvas that resample_kernel<true> filled (the unnormalised resampled
// kernel), for the ring means of the Split look.
__global__ void __launch_bounds__(256) ring_sums_kernel(PsfBankArgs a) {
    stream_order();
    __shared__ float ring[kRingSpanTall];
    const int b = blockIdx.z;
    const int K = a.K, R = a.R;
    const int tx0 = blockIdx.x * kTile, ty0 = blockIdx.y * kTallH;
    const int tid = threadIdx.x + threadIdx.y * 32;
    const int rbase = tile_ring_base(tx0, ty0, R, R, kTallH);
    for (int i = tid; i < kRingSpanTall; i += 256) ring[i] = 0.0f;
    __syncthreads();
    const float kc = static_cast<float>(K - 1) * 0.5f;
    const float* canvas = a.canvas + static_cast<size_t>(b) * K * K;
    const int x = tx0 + threadIdx.x;
    const float dx = static_cast<float>(x) - kc;
    for (int i = 0; i < kTallH / 8; ++i) {
        const int y = ty0 + threadIdx.y + 8 * i;
        if (y >= K) break;  // uniform: a warp is one canvas row
        float v = 0.0f;
        int slot = -1;
        if (x < K) {
            const float dy = static_cast<float>(y) - kc;
            v = __ldg(canvas + static_cast<size_t>(y) * K + x);
            slot = min(R, static_cast<int>(roundf(sqrtf(dx * dx + dy * dy)))) - rbase;
        }
        warp_runs_accumulate<false>(slot, v, v, ring, nullptr);
    }
    __syncthreads();
    const size_t ro = static_cast<size_t>(b) * (R + 1);
    for (int i = tid; i < kRingSpanTall; i += 256)
        if (ring[i] != 0.0f && rbase + i <= R) atomicAdd(&a.ring_round[ro + rbase + i], static_cast<double>(ring[i]));
}

// grid (ceil(K/32), ceil(K/128), B): shaped kernel (reshapeAnisotropy of the
// base kernel against its azimuthal mean, LensDiffCpuReference.cpp:1088-1135)
// written in place, its sum, and its ring energy / peak by ceil(r)
// (estimateAdaptiveSupportRadius, :984-1007).
__global__ void __launch_bounds__(256) shape_stats_kernel(PsfBankArgs a) {
    stream_order();
    __shared__ float ring_e[kRingSpanTall];
    __shared__ unsigned int ring_p[kRingSpanTall];
    __shared__ float mean_r[kRingSpanTall];
    const int b = blockIdx.z;
    const int tid = threadIdx.x + threadIdx.y * 32;
    const double s1 = a.scalars[b].s1;
    const int K = a.K, R = a.R;
    const int tx0 = blockIdx.x * kTile, ty0 = blockIdx.y * kTallH;
    const int rbase = tile_ring_base(tx0, ty0, R, R, kTallH);
    // ring means (round(r) rings) the tile can touch
    const float* rm = a.ring_mean + static_cast<size_t>(b) * (R + 1);
    for (int i = tid; i < kRingSpanTall; i += 256) {
        ring_e[i] = 0.0f;
        ring_p[i] = 0u;
        const int r = rbase + i;
        mean_r[i] = r <= R ? rm[r] : 0.0f;
    }
    __syncthreads();
    const float inv_s1 = static_cast<float>(1.0 / s1);
    const float gain = a.gain;
    const float kc = static_cast<float>(K - 1) * 0.5f;
    float* canvas = a.canvas + static_cast<size_t>(b) * K * K;
    float lsum = 0.0f;  // this thread's pixels; one double add per thread below
    unsigned int lpeak = 0u;
    const int x = tx0 + threadIdx.x;
    // the thread's four canvas reads are issued before any is used (each
    // element is read, then written, by this thread only)
    float raw[kTallH / 8];
#pragma unroll
    for (int i = 0; i < kTallH / 8; ++i) {
        const int y = ty0 + threadIdx.y + 8 * i;
        raw[i] = (x < K && y < K) ? __ldg(canvas + static_cast<size_t>(y) * K + x) : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < kTallH / 8; ++i) {
        const int y = ty0 + threadIdx.y + 8 * i;
        const bool in = x < K && y < K;
        float v = 0.0f;
        int slot = -1;
        if (in) {
            const float dx = static_cast<float>(x) - kc;
            const float dy = static_cast<float>(y) - kc;
            const float rad = sqrtf(dx * dx + dy * dy);
            const size_t idx = static_cast<size_t>(y) * K + x;
            const float base = raw[i] * inv_s1;
            const float mean = mean_r[min(R, static_cast<int>(roundf(rad))) - rbase];
            v = fmaxf(0.0f, mean + (base - mean) * gain);
            canvas[idx] = v;
            lsum += v;
            lpeak = max(lpeak, __float_as_uint(v));
            slot = min(R, static_cast<int>(ceilf(rad))) - rbase;
        }
        warp_runs_accumulate<true>(slot, v, v, ring_e, ring_p);
    }
    __syncthreads();
    const size_t ro = static_cast<size_t>(b) * (R + 1);
    for (int i = tid; i < kRingSpanTall; i += 256) {
        if (rbase + i <= R) {
            if (ring_e[i] != 0.0f) atomicAdd(&a.ring_ceil[ro + rbase + i], static_cast<double>(ring_e[i]));
            if (ring_p[i] != 0u) atomicMax(&a.ring_peak[ro + rbase + i], ring_p[i]);
        }
    }
    for (int o = 16; o > 0; o >>= 1) lpeak = max(lpeak, __shfl_xor_sync(0xffffffffu, lpeak, o));
    if ((tid & 31) == 0 && lpeak != 0u) atomicMax(&a.scalars[b].peak, lpeak);
    const double tot = block_sum(static_cast<double>(lsum));
    if (tid == 0) atomicAdd(&a.scalars[b].s3, tot);
}

// grid (B), block 256: adaptive support radius and taper constants
// (estimateAdaptiveSupportRadius :1009-1030, paddedAdaptiveSupportRadius
// :1033-1036, cropKernelToRadius :1039, applySupportBoundaryTaper :962-965).
// Suffix maxima of the ring peaks and prefix sums of the ring energies are
// block scans over per-thread chunks of rings.
__global__ void __launch_bounds__(256) support_kernel(PsfBankArgs a) {
    stream_order();
    __shared__ float chunk_max[256];
    __shared__ double chunk_sum[256];
    __shared__ int first_hit;
    const int b = blockIdx.x;
    const int tid = threadIdx.x;
    PsfScalars& sc = a.scalars[b];
    const int R = a.R;
    const int rm = min(R, a.K / 2);
    const int nr = rm + 1;
    const int per = (nr + 255) / 256;
    const int r0 = tid * per, r1 = min(nr, r0 + per);
    const double* e = a.ring_ceil + static_cast<size_t>(b) * (R + 1);
    const unsigned int* pk = a.ring_peak + static_cast<size_t>(b) * (R + 1);
    const double total = sc.s3;
    const float peak = __uint_as_float(sc.peak);
    float lmax = 0.0f;
    double lsum = 0.0;
    for (int r = r0; r < r1; ++r) {
        lmax = fmaxf(lmax, __uint_as_float(pk[r]));
        lsum += e[r];
    }
    chunk_max[tid] = lmax;
    chunk_sum[tid] = lsum;
    if (tid == 0) first_hit = 1 << 30;
    __syncthreads();
    {  // exclusive prefix sums / suffix maxima over the 256 chunks: one warp, eight chunks a lane
        if (tid < 32) {
            double run = 0.0, sums[8];
            float m = 0.0f, maxs[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                sums[i] = run;
                run += chunk_sum[tid * 8 + i];
                maxs[7 - i] = m;  // maximum over this lane's chunks after 7 - i
                m = fmaxf(m, chunk_max[tid * 8 + 7 - i]);
            }
            double before = run;
            float after = m;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double t = __shfl_up_sync(0xffffffffu, before, o);
                const float u = __shfl_down_sync(0xffffffffu, after, o);
                if (tid >= o) before += t;
                if (tid + o < 32) after = fmaxf(after, u);
            }
            before -= run;
            after = __shfl_down_sync(0xffffffffu, after, 1);
            if (tid == 31) after = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                chunk_sum[tid * 8 + i] = before + sums[i];
                chunk_max[tid * 8 + i] = fmaxf(after, maxs[i]);
            }
        }
    }
    __syncthreads();
    // the normalised kernel has total 1 and peak = peak / total
    const bool degenerate = !(total > 0.0) || (static_cast<double>(peak) / total <= 1e-6);
    if (!degenerate && r0 < r1) {
        // suffix maxima inside this chunk, then the first ring that passes
        float suffix[64];
        const int len = r1 - r0;  // <= 64 for R <= 16383
        float m = chunk_max[tid];
        for (int k = len - 1; k >= 0; --k) {
            suffix[k] = m;  // maximum over rings > r0 + k
            m = fmaxf(m, __uint_as_float(pk[r0 + k]));
        }
        double cum = chunk_sum[tid];
        const double thr_cap = static_cast<double>(0.9999f);
        const float thr_peak = peak * 2e-4f;
        for (int k = 0; k < len; ++k) {
            cum += e[r0 + k];
            if (cum / total >= thr_cap && suffix[k] <= thr_peak) {
                atomicMin(&first_hit, r0 + k);
                break;
            }
        }
    }
    __syncthreads();
    if (tid != 0) return;
    int est = max(4, rm);
    if (!degenerate && first_hit < (1 << 30)) est = max(4, first_hit + 1);
    const int pad = max(6, min(24, static_cast<int>(ceilf(static_cast<float>(max(1, est)) * 0.05f))));
    int rho = min(max(est + pad, 4), max(4, R));
    rho = min(max(rho, 1), a.K / 2);
    sc.radius = rho;
    const float extent = fmaxf(1.0f, static_cast<float>(rho));
    const float fade = fmaxf(6.0f, fminf(24.0f, extent * 0.04f));
    sc.extent = extent;
    sc.fade = fade;
    sc.start = fmaxf(0.0f, extent - fade);
}

// grid (ceil((R+1)/16), B), block 256: s4 = sum over the crop box of taper *
// normalised shaped kernel, the normaliser of cropKernelToRadius and
// applySupportBoundaryTaper (LensDiffCpuReference.cpp:1038-1058, :957-982).
// The canvas keeps the shaped kernel; the crop and the taper are applied
// where the kernel is read (combine_kernel, split_sums_kernel, export_kernel).
// The taper is 1 up to radius `start` and 0 from `extent` on, and every pixel
// with r < extent lies in the crop box, so s4 = (the ceil(r) ring energies of
// rings 0 .. S0 = floor(start)) / s3 + the annulus S0 < r < extent pixel by
// pixel.  A pixel's ring is ceil(sqrtf(dx^2 + dy^2)) <= S0 exactly when
// dx^2 + dy^2 <= S0^2 (integers; exact below 2^24), and its taper is 0 from
// dx^2 + dy^2 = rho^2 on (extent = rho), so each row of the quadrant dx, dy >=
// 0 reads only the dx between, with the mirror images, which share the
// pixel's taper.  A warp takes two quadrant rows, a CTA's reductions serve 16
// (a row a warp of the whole crop box, out to its corners: 33 us for 31
// wavelengths at K = 1025, 14 us now).
constexpr int kCropRows = 16;

__device__ __forceinline__ int isqrt_floor(int v) {  // floor(sqrt(v)), v >= 0
    int r = static_cast<int>(sqrtf(static_cast<float>(v)));
    while (r > 0 && r * r > v) --r;
    while ((r + 1) * (r + 1) <= v) ++r;
    return r;
}

__global__ void __launch_bounds__(256) crop_sum_kernel(PsfBankArgs a) {
    stream_order();
    const int b = blockIdx.y;
    const PsfScalars& sc = a.scalars[b];
    const int rho = sc.radius;
    const int K = a.K, R = a.R;
    const int d0 = static_cast<int>(blockIdx.x) * kCropRows;
    if (d0 > rho) return;  // uniform
    const float inv_s3 = static_cast<float>(1.0 / sc.s3);
    const float extent = sc.extent, fade = sc.fade, start = sc.start;
    const int s0 = static_cast<int>(floorf(start));
    const int lane = threadIdx.x & 31;
    const float* centre = a.canvas + static_cast<size_t>(b) * K * K + static_cast<size_t>(R) * K + R;
    float lsum = 0.0f;
    for (int i = 0; i < kCropRows / 8; ++i) {
        const int dy = d0 + static_cast<int>(threadIdx.x >> 5) + 8 * i;
        if (dy > rho) break;  // uniform: a warp walks rows
        const int in2 = s0 * s0 - dy * dy;
        const int first = in2 >= 0 ? isqrt_floor(in2) + 1 : 0;
        const int last = isqrt_floor(rho * rho - dy * dy);
        const float* up = centre + static_cast<ptrdiff_t>(dy) * K;
        const float* down = centre - static_cast<ptrdiff_t>(dy) * K;
        const float dy2 = static_cast<float>(dy) * static_cast<float>(dy);
        for (int dx = first + lane; dx <= last; dx += 32) {
            float v = __ldg(up + dx);
            if (dx > 0) v += __ldg(up - dx);
            if (dy > 0) {
                v += __ldg(down + dx);
                if (dx > 0) v += __ldg(down - dx);
            }
            const float x = static_cast<float>(dx);
            lsum += (v * inv_s3) * taper_weight(sqrtf(x * x + dy2), extent, fade, start);
        }
    }
    double tot = block_sum(static_cast<double>(lsum));
    if (blockIdx.x == 0) {  // the rings inside the taper's flat part
        const double* e = a.ring_ceil + static_cast<size_t>(b) * (R + 1);
        double ring = 0.0;
        for (int r = threadIdx.x; r <= s0; r += blockDim.x) ring += e[r];
        ring = block_sum(ring);
        if (threadIdx.x == 0) tot += ring / sc.s3;
    }
    if (threadIdx.x == 0) atomicAdd(&a.scalars[b].s4, tot);
}

// grid (ceil(K/32), ceil(K/32), B): the Split look's normalisers after the
// crop (the canvas holds the shaped kernel; taper applied here):
// s_core = sum of mean * taper, s_struct = sum of max(0, shaped * taper / s3
// - mean * taper) over the crop box.
__global__ void __launch_bounds__(256) split_sums_kernel(PsfBankArgs a) {
    stream_order();
    const int b = blockIdx.z;
    const PsfScalars& sc = a.scalars[b];
    const float inv_s3 = static_cast<float>(1.0 / sc.s3);
    const int rho = sc.radius;
    const int K = a.K, R = a.R;
    const float* canvas = a.canvas + static_cast<size_t>(b) * K * K;
    const float* rm = a.ring_mean + static_cast<size_t>(b) * (R + 1);
    const int x = blockIdx.x * kTile + threadIdx.x;
    double lcore = 0.0, lstruct = 0.0;
#pragma unroll
    for (int i = 0; i < kTile / 8; ++i) {
        const int y = blockIdx.y * kTile + threadIdx.y + 8 * i;
        if (x < K && y < K) {
            const int ix = x - R, iy = y - R;
            if (abs(ix) <= rho && abs(iy) <= rho) {
                const float dx = static_cast<float>(ix), dy = static_cast<float>(iy);
                const float rad = sqrtf(dx * dx + dy * dy);
                const float wgt = taper_weight(rad, sc.extent, sc.fade, sc.start);
                const float mt = rm[min(R, static_cast<int>(roundf(rad)))] * wgt;
                lcore += static_cast<double>(mt);
                lstruct += static_cast<double>(fmaxf(0.0f, (canvas[static_cast<size_t>(y) * K + x] * wgt) * inv_s3 - mt));
            }
        }
    }
    const double tc = block_sum(lcore);
    if (threadIdx.x == 0 && threadIdx.y == 0) atomicAdd(&a.scalars[b].s_core, tc);
    __syncthreads();
    const double ts = block_sum(lstruct);
    if (threadIdx.x == 0 && threadIdx.y == 0) atomicAdd(&a.scalars[b].s_struct, ts);
}

// grid (ceil((R+1)/32), ceil((R+1)/8)), block (32, 8): out[k] = sum_b
// coef[k][b] * final_b with final_b = crop_b(canvas_b * taper_b) / (s3_b *
// s4_b): the crop box and boundary taper of each wavelength
// (cropKernelToRadius, applySupportBoundaryTaper,
// LensDiffCpuReference.cpp:1038-1058, :957-982) are applied here as the shaped
// kernels are read.  A thread takes a pixel of the quadrant dx, dy >= 0 and its
// mirror images, which share the radius, the crop test and the taper of every
// wavelength; kL wavelengths' reads are issued before any is used; per pixel
// the wavelengths are summed in order.  31 wavelengths at K = 1025 take 38 us
// (reading the canvases takes 20 of HBM time; 67 us with four unrelated
// pixels a thread).  SPLIT: the core and structure kernels of the Split look
// instead: core = mean * taper / s_core, structure = max(0, shaped * taper /
// s3 - mean * taper) / s_struct.
struct CombineBin {
    float w[4];                     // coef[k][b] / (s3 s4), Split: coef[k][b]
    float ext, fade, start;         // taper
    int rho;                        // crop radius
    float inv_s3, inv_core, inv_struct;
};

// NK: output kernels (1 Mono, 3 spectral, 4 with the luma lock; Split: 4).
template <bool SPLIT, int NK>
__global__ void __launch_bounds__(256) combine_kernel(CombineArgs a) {
    stream_order();
    __shared__ CombineBin bin[kMaxBins];
    const int tid = threadIdx.x + threadIdx.y * 32;
    const int B = a.bank.B;
    for (int b = tid; b < B; b += 256) {
        const PsfScalars& sc = a.bank.scalars[b];
        CombineBin& t = bin[b];
        const float ib = SPLIT ? 1.0f : static_cast<float>(1.0 / (sc.s3 * sc.s4));
        for (int k = 0; k < 4; ++k) t.w[k] = a.coef[k][b] * ib;
        t.ext = sc.extent;
        t.fade = sc.fade;
        t.start = sc.start;
        t.rho = sc.radius;
        t.inv_s3 = static_cast<float>(1.0 / sc.s3);
        t.inv_core = sc.s_core > 0.0 ? static_cast<float>(1.0 / sc.s_core) : 0.0f;
        t.inv_struct = sc.s_struct > 0.0 ? static_cast<float>(1.0 / sc.s_struct) : 0.0f;
    }
    __syncthreads();
    const int K = a.bank.K, R = a.bank.R;
    const int ix = blockIdx.x * 32 + threadIdx.x, iy = blockIdx.y * 8 + threadIdx.y;
    if (ix > R || iy > R) return;
    const size_t plane = static_cast<size_t>(K) * K;
    constexpr int kP = 4;  // the mirror images (on an axis some coincide: the same value, written twice)
    const int up = (R + iy) * K + R, down = (R - iy) * K + R;
    const int idx[kP] = {up + ix, up - ix, down + ix, down - ix};
    const int aix = max(ix, iy);  // inside the crop box of b iff aix <= rho[b]
    const float dx = static_cast<float>(ix), dy = static_cast<float>(iy);
    const float rad = sqrtf(dx * dx + dy * dy);
    constexpr int kL = 4;
    if constexpr (!SPLIT) {
        float acc[kP][NK] = {};
        for (int b0 = 0; b0 < B; b0 += kL) {
            float v[kL][kP];
#pragma unroll
            for (int l = 0; l < kL; ++l) {
                const int b = min(b0 + l, B - 1);
                const bool in = b0 + l < B && aix <= bin[b].rho;
                const float* cv = a.bank.canvas + b * plane;
#pragma unroll
                for (int p = 0; p < kP; ++p) v[l][p] = in ? __ldg(cv + idx[p]) : 0.0f;
            }
#pragma unroll
            for (int l = 0; l < kL; ++l) {
                if (b0 + l >= B) break;
                const CombineBin& cb = bin[b0 + l];
                if (aix > cb.rho) continue;
                const float wgt = taper_weight(rad, cb.ext, cb.fade, cb.start);
#pragma unroll
                for (int p = 0; p < kP; ++p) {
                    const float f = v[l][p] * wgt;
#pragma unroll
                    for (int k = 0; k < NK; ++k) acc[p][k] += cb.w[k] * f;
                }
            }
        }
#pragma unroll
        for (int p = 0; p < kP; ++p) {
#pragma unroll
            for (int k = 0; k < NK; ++k) a.out[k * plane + idx[p]] = acc[p][k];
        }
    } else {
        const int ring = min(R, static_cast<int>(roundf(rad)));
        float core[4] = {}, strc[kP][4] = {};
        for (int b0 = 0; b0 < B; b0 += kL) {
            float v[kL][kP], mean[kL];
#pragma unroll
            for (int l = 0; l < kL; ++l) {
                const int b = min(b0 + l, B - 1);
                const bool in = b0 + l < B && aix <= bin[b].rho;
                const float* cv = a.bank.canvas + b * plane;
                mean[l] = in ? __ldg(a.bank.ring_mean + static_cast<size_t>(b) * (R + 1) + ring) : 0.0f;
#pragma unroll
                for (int p = 0; p < kP; ++p) v[l][p] = in ? __ldg(cv + idx[p]) : 0.0f;
            }
#pragma unroll
            for (int l = 0; l < kL; ++l) {
                if (b0 + l >= B) break;
                const CombineBin& cb = bin[b0 + l];
                if (aix > cb.rho) continue;
                const float wgt = taper_weight(rad, cb.ext, cb.fade, cb.start);
                const float mt = mean[l] * wgt;
                const float c = mt * cb.inv_core;
#pragma unroll
                for (int k = 0; k < 4; ++k) core[k] += cb.w[k] * c;
#pragma unroll
                for (int p = 0; p < kP; ++p) {
                    const float st = fmaxf(0.0f, (v[l][p] * wgt) * cb.inv_s3 - mt) * cb.inv_struct;
#pragma unroll
                    for (int k = 0; k < 4; ++k) strc[p][k] += cb.w[k] * st;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k >= a.n_ker) break;
#pragma unroll
            for (int p = 0; p < kP; ++p) {
                a.out[k * plane + idx[p]] = core[k];
                a.out[(a.n_ker + k) * plane + idx[p]] = strc[p][k];
            }
        }
    }
}

// grid (ceil(K/32), ceil(K/32), B): final kernels packed at offsets[b].
__global__ void __launch_bounds__(256) export_kernel(PsfBankArgs a, const int64_t* offsets, float* out) {
    const int b = blockIdx.z;
    const PsfScalars& sc = a.scalars[b];
    const int rho = sc.radius;
    const int side = 2 * rho + 1;
    const float inv = static_cast<float>(1.0 / (sc.s3 * sc.s4));
    const float* canvas = a.canvas + static_cast<size_t>(b) * a.K * a.K;
    const int x = blockIdx.x * kTile + threadIdx.x;
    for (int i = 0; i < kTile / 8; ++i) {
        const int y = blockIdx.y * kTile + threadIdx.y + 8 * i;
        if (x >= a.K || y >= a.K) continue;
        const int ix = x - a.R + rho, iy = y - a.R + rho;
        if (ix < 0 || iy < 0 || ix >= side || iy >= side) continue;
        const float dx = static_cast<float>(x - a.R), dy = static_cast<float>(y - a.R);
        const float wgt = taper_weight(sqrtf(dx * dx + dy * dy), sc.extent, sc.fade, sc.start);
        out[offsets[b] + static_cast<int64_t>(iy) * side + ix] = (canvas[static_cast<size_t>(y) * a.K + x] * wgt) * inv;
    }
}

// ---- first-minimum calibration ------------------------------------------------------
// grid (ceil(S/32), ceil(S/32)), block (32, 8): sums and counts of the shifted
// intensity by round(r) around shiftedSpectrumCenterCoordinate.
// The window psf[y * stride + x], x, y < n, is the square of the shifted PSF
// starting at (x0, x0); total == null: the caller supplies the full PSF's sum.
__global__ void __launch_bounds__(256) profile_kernel(const float* psf, int stride, int n, int x0, int S,
                                                      double* sums, int* counts, double* total) {
    __shared__ double rs[kRingSpan];
    __shared__ int rc[kRingSpan];
    const int tid = threadIdx.x + threadIdx.y * 32;
    const float c = (S & 1) == 0 ? static_cast<float>(S) * 0.5f : static_cast<float>(S - 1) * 0.5f;
    const int ci = static_cast<int>(c);
    const int rmax = S / 2;
    const int tx0 = blockIdx.x * kTile, ty0 = blockIdx.y * kTile;
    const int rbase = tile_ring_base(x0 + tx0, x0 + ty0, ci, rmax);
    for (int i = tid; i < kRingSpan; i += 256) {
        rs[i] = 0.0;
        rc[i] = 0;
    }
    __syncthreads();
    double lsum = 0.0;
    const int x = tx0 + threadIdx.x;
    for (int i = 0; i < kTile / 8; ++i) {
        const int y = ty0 + threadIdx.y + 8 * i;
        if (x < n && y < n) {
            const float dx = static_cast<float>(x0 + x) - c;
            const float dy = static_cast<float>(x0 + y) - c;
            const int r = min(rmax, static_cast<int>(roundf(sqrtf(dx * dx + dy * dy))));
            const float v = psf[static_cast<size_t>(y) * stride + x];
            lsum += v;
            atomicAdd(&rs[r - rbase], static_cast<double>(v));
            atomicAdd(&rc[r - rbase], 1);
        }
    }
    __syncthreads();
    for (int i = tid; i < kRingSpan; i += 256) {
        if (rc[i] != 0 && rbase + i <= rmax) {
            atomicAdd(&sums[rbase + i], rs[i]);
            atomicAdd(&counts[rbase + i], rc[i]);
        }
    }
    if (total) {
        const double tot = block_sum(lsum);
        if (tid == 0) atomicAdd(total, tot);
    }
}

__device__ float refine_parabolic(double l, double c, double r) {
    const double den = l - 2.0 * c + r;
    if (fabs(den) < 1e-6) return 0.0f;
    return static_cast<float>(fmin(fmax(0.5 * (l - r) / den, -0.5), 0.5));
}

// One thread: radialMeanProfile normalised by the total, [1,2,1]/4 smoothing,
// first local minimum after >= 2 descents with parabolic refinement, fallback
// argmin over [1, max(4, S/8)] (LensDiffCpuReference.cpp:897-955).
// n: rings profiled (S / 2 + 1 for the whole PSF); truncated: the rings past
// n exist but were not profiled, so a scan that finds no minimum inside them
// reports r0 = -1 instead of taking the fallback over all rings.
__global__ void first_zero_scan_kernel(const double* sums, const int* counts, const double* total, int S, int n,
                                       int truncated, double* prof, float* r0) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double t = *total > 0.0 ? *total : 1.0;
    for (int r = 0; r < n; ++r) prof[r] = (sums[r] / t) / max(1, counts[r]);
    if (n < 4) {
        *r0 = 1.0f;
        return;
    }
    double* sm = prof + n;
    for (int i = 0; i < n; ++i) {
        const double left = prof[i == 0 ? 0 : i - 1];
        const double right = prof[i + 1 < n ? i + 1 : i];
        sm[i] = (left + 2.0 * prof[i] + right) * 0.25;
    }
    int best = 1;
    double bestv = sm[1];
    int desc = sm[1] < sm[0] ? 1 : 0;
    for (int i = 2; i + 1 < n; ++i) {
        if (sm[i] <= sm[i - 1]) {
            desc += 1;
            if (sm[i] < bestv) {
                bestv = sm[i];
                best = i;
            }
            continue;
        }
        if (desc >= 2 && best > 0 && best + 1 < n) {
            *r0 = fmaxf(1.0f, static_cast<float>(best) + refine_parabolic(sm[best - 1], sm[best], sm[best + 1]));
            return;
        }
        best = i;
        bestv = sm[i];
        desc = 0;
    }
    if (truncated) {
        *r0 = -1.0f;
        return;
    }
    const int limit = max(2, min(n - 1, max(4, S / 8)));
    best = 1;
    bestv = sm[1];
    for (int i = 2; i <= limit; ++i) {
        if (sm[i] < bestv) {
            bestv = sm[i];
            best = i;
        }
    }
    if (best > 0 && best + 1 < n)
        *r0 = fmaxf(1.0f, static_cast<float>(best) + refine_parabolic(sm[best - 1], sm[best], sm[best + 1]));
    else
        *r0 = static_cast<float>(best);
}

// scale * sum of the squared pupil amplitude: by Parseval, the sum of the
// unnormalised S x S PSF when scale = S^2.
__global__ void __launch_bounds__(256) pupil_energy_kernel(PsfBankArgs a, double scale, double* out) {
    const int n = a.pupil.size * a.pupil.size;
    double acc = 0.0;
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        const float amp = a.pupil_pre[i].x;
        acc += static_cast<double>(amp) * amp;
    }
    const double t = block_sum(acc);
    if (threadIdx.x == 0) atomicAdd(out, t * scale);
}

__global__ void normalize_psf_kernel(float* psf, int64_t n, const PsfScalars* sc) {
    const double e = sc->energy;
    const float inv = e > 0.0 ? static_cast<float>(1.0 / e) : 1.0f;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        psf[i] *= inv;
}

// ---- launch helpers ---------------------------------------------------------------
// Row pass: one length-S transform per CTA.  Column pass: C adjacent window
// columns per CTA, C = 4 / 2 / 1 for S <= 2048 / 4096 / larger (S * C <= 8192
// keeps the E = 25 family up to S = 4096).
template <int E>
void rows_launch(const PsfBankArgs& a, cudaStream_t s) {
    dim3 grid(a.row_n, a.B);
    launch_after(psf_rows_kernel<E>, grid, fft_threads(a.S, 1, E), a.S * sizeof(float2), s, a);
}

template <int E, int C>
void cols_launch(const PsfBankArgs& a, cudaStream_t s) {
    dim3 grid((a.win_stride + C - 1) / C, a.B);
    launch_after(psf_cols_kernel<E, C>, grid, fft_threads(a.S, C, E), static_cast<size_t>(a.S) * C * sizeof(float2), s,
                 a);
}

dim3 tall_grid(const PsfBankArgs& a) {
    return dim3((a.K + kTile - 1) / kTile, (a.K + kTallH - 1) / kTallH, a.B);
}

dim3 canvas_grid(const PsfBankArgs& a, int z) {
    return dim3((a.K + kTile - 1) / kTile, (a.K + kTile - 1) / kTile, z);
}

template <class Kern>
void opt_in(Kern k, size_t bytes) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

}  // namespace

void launch_pupil_pre(const PsfBankArgs& a, cudaStream_t s) {
    const int n = a.pupil.size * a.pupil.size;
    launch_after(pupil_pre_kernel, (n + 255) / 256, 256, 0, s, a);
}

void launch_psf_rows(const PsfBankArgs& a, cudaStream_t s) {
    if (fft_family(a.S, 1) == kE25) rows_launch<kE25>(a, s);
    else rows_launch<kE16>(a, s);
}

void launch_psf_cols(const PsfBankArgs& a, cudaStream_t s) {
    if (a.S <= 2048) cols_launch<kE25, 4>(a, s);
    else if (a.S <= 4096) cols_launch<kE25, 2>(a, s);
    else if (fft_family(a.S, 1) == kE25) cols_launch<kE25, 1>(a, s);
    else cols_launch<kE16, 1>(a, s);
}

bool fused_shaping(const PsfBankArgs& a) { return a.gain == 1.0f; }

// filtered: some wavelength is box-filtered; inv_max: the largest sample
// distance of the others (0: none).
// Filtered tiles: 32 rows, or 16 where 128-row tiles would not give every SM
// one CTA.  The canvas under a box filter reaches far outside the PSF, where
// its pixels are zero, so only the central tiles have work and short ones
// spread it: 128 / 64 / 32 / 16 / 8 rows took 197 / 70 / 69 / 78 / 100 us for
// 16 wavelengths at K = 513, 73 / 24 / 26 / 16 / 14 us for 3 at K = 257.
// Quadrant tiles: 128 rows (112 us for 31 wavelengths at K = 1025 and
// inv_scale <= 0.40, 118 us with 64), 64 where the staged boxes of 128 rows
// would take over 25 KB and cost resident CTAs (inv_max > 0.5), 16 where 64
// rows would not give every SM two CTAs.
void launch_resample(const PsfBankArgs& a, bool filtered, float inv_max, cudaStream_t s) {
    const dim3 tall = tall_grid(a);
    if (filtered && a.h16) {
        if (fused_shaping(a)) launch_after(resample_tile_kernel<true>, tall, dim3(32, 8), 0, s, a);
        else launch_after(resample_tile_kernel<false>, tall, dim3(32, 8), 0, s, a);
        return;
    }
    ResampleGrid g{};
    size_t sm = 0;
    int grid = 0;
    if (inv_max > 0.0f) {
        g.qx = (a.R + kTile) / kTile;
        g.qth = g.qx * ((a.R + 64) / 64) * a.B < 2 * 148 ? 16 : (inv_max <= 0.5f ? kQuadH : 64);
        g.qy = (a.R + g.qth) / g.qth;
        g.sw = quad_stage(kTile, inv_max);
        g.sh = quad_stage(g.qth, inv_max);
        g.nq = g.qx * g.qy * a.B;
        sm = kQuadRingBytes + 4 * sizeof(float) * g.sw * g.sh;
        grid = g.nq;
    }
    if (filtered) {
        g.fth = tall.x * tall.y * tall.z < 148 ? 16 : kTile;
        g.fx = tall.x;
        g.fy = (a.K + g.fth - 1) / g.fth;
        sm = std::max(sm, sizeof(FilterSmem));
        grid += g.fx * g.fy * a.B;
    }
    if (fused_shaping(a)) launch_after(resample_kernel<true>, grid, dim3(32, 8), sm, s, a, g);
    else launch_after(resample_kernel<false>, grid, dim3(32, 8), sm, s, a, g);
}

void launch_shape_stats(const PsfBankArgs& a, cudaStream_t s) {
    launch_after(ring_mean_kernel, a.B, 256, 0, s, a);
    launch_after(shape_stats_kernel, tall_grid(a), dim3(32, 8), 0, s, a);
}

void launch_ring_means(const PsfBankArgs& a, cudaStream_t s) {
    launch_after(ring_sums_kernel, tall_grid(a), dim3(32, 8), 0, s, a);
    launch_after(ring_mean_kernel, a.B, 256, 0, s, a);
}

void launch_support(const PsfBankArgs& a, cudaStream_t s) { launch_after(support_kernel, a.B, 256, 0, s, a); }

void launch_crop_sum(const PsfBankArgs& a, cudaStream_t s) {
    launch_after(crop_sum_kernel, dim3((a.R + kCropRows) / kCropRows, a.B), 256, 0, s, a);
}

void launch_split_sums(const PsfBankArgs& a, cudaStream_t s) {
    launch_after(split_sums_kernel, canvas_grid(a, a.B), dim3(32, 8), 0, s, a);
}

void launch_combine(const CombineArgs& a, cudaStream_t s) {
    const dim3 grid((a.bank.R + 32) / 32, (a.bank.R + 8) / 8), block(32, 8);
    if (a.split) launch_after(combine_kernel<true, 4>, grid, block, 0, s, a);
    else if (a.n_ker == 1) launch_after(combine_kernel<false, 1>, grid, block, 0, s, a);
    else if (a.n_ker == 3) launch_after(combine_kernel<false, 3>, grid, block, 0, s, a);
    else launch_after(combine_kernel<false, 4>, grid, block, 0, s, a);
}

void launch_export(const PsfBankArgs& a, const int64_t* offsets_dev, float* out, cudaStream_t s) {
    export_kernel<<<canvas_grid(a, a.B), dim3(32, 8), 0, s>>>(a, offsets_dev, out);
}

void launch_first_zero(const float* psf, int S, double* ring_sums, int* ring_counts, double* total, float* r0_out,
                       cudaStream_t s) {
    launch_first_zero_window(psf, S, S, 0, S, S / 2 + 1, ring_sums, ring_counts, total, true, r0_out, s);
}

void launch_first_zero_window(const float* psf, int stride, int n, int x0, int S, int rings, double* ring_sums,
                              int* ring_counts, double* total, bool own_total, float* r0_out, cudaStream_t s) {
    dim3 grid((n + kTile - 1) / kTile, (n + kTile - 1) / kTile);
    profile_kernel<<<grid, dim3(32, 8), 0, s>>>(psf, stride, n, x0, S, ring_sums, ring_counts,
                                                own_total ? total : nullptr);
    // profile scratch follows the ring sums: 2 * (S/2 + 1) doubles
    first_zero_scan_kernel<<<1, 32, 0, s>>>(ring_sums, ring_counts, total, S, rings, rings < S / 2 + 1 ? 1 : 0,
                                            ring_sums + (S / 2 + 1), r0_out);
}

void launch_pupil_energy(const PsfBankArgs& a, double scale, double* out, cudaStream_t s) {
    pupil_energy_kernel<<<64, 256, 0, s>>>(a, scale, out);
}

void launch_normalize_psf(float* psf, int n, const PsfScalars* sc, cudaStream_t s) {
    normalize_psf_kernel<<<592, 256, 0, s>>>(psf, static_cast<int64_t>(n), sc);
}

void configure_psf_kernels() {
    const size_t quad = kQuadRingBytes + 4 * sizeof(float) * quad_stage(kTile, 1.0f) * quad_stage(64, 1.0f);
    opt_in(resample_kernel<true>, quad);
    opt_in(resample_kernel<false>, quad);
    opt_in(psf_rows_kernel<kE25>, 12800 * 8);
    opt_in(psf_rows_kernel<kE16>, 16384 * 8);
    opt_in(psf_cols_kernel<kE25, 4>, 2048 * 4 * 8);
    opt_in(psf_cols_kernel<kE25, 2>, 4096 * 2 * 8);
    opt_in(psf_cols_kernel<kE25, 1>, 12800 * 8);
    opt_in(psf_cols_kernel<kE16, 1>, 16384 * 8);
}

}  // namespace ld
