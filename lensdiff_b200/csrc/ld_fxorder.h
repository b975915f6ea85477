// ld_fxorder.h — the stage order of the FP16 form's transforms.
//
// The FP16 form stores row spectra, kernel spectra and column outputs as half.
// Two radix orders of one transform round their FP32 sums differently, and
// after the rounding to half about one stored value in a hundred then falls to
// its neighbour: 0.05 to 0.15 of the form's own error, up to 5e-5 of a small
// log-encoded frame.  So its compiled passes run the stages of the
// runtime-planned transform (ld_fft.cuh) with the same twiddles, in the same
// order, and give its bits; two neighbouring stages that are small are taken
// together in registers, which leaves three passes over shared memory for
// nearly every length.  The FP32 form and the passes that end in FP32 keep the
// faster orders of ld_fxplans.h.
#pragma once

#include <cuda_runtime.h>

namespace ld {

// The radices of the runtime-planned transform of length n, first stage
// first (kPlanRadices' order); returns how many, 0 when n is not 5-smooth.
// Pairs of fives are 25 (where allowed: the 25-element family), fours of twos
// 16, the rest 8 / 4 / 2 (16 * 2 becomes 8 * 4), threes 3.
constexpr int plan_radices(int n, bool allow25, int (&out)[16]) {
    int m = n, twos = 0, threes = 0, fives = 0, k = 0;
    if (n < 2) return 0;
    for (; m % 2 == 0; m /= 2) ++twos;
    for (; m % 3 == 0; m /= 3) ++threes;
    for (; m % 5 == 0; m /= 5) ++fives;
    if (m != 1) return 0;
    int q16 = twos / 4;
    const int rem = twos % 4;
    const bool eight_four = rem == 1 && q16 > 0;
    if (eight_four) --q16;
    if ((allow25 ? fives / 2 + fives % 2 : fives) + threes + q16 + 2 > 16) return 0;
    if (allow25)
        for (; fives >= 2; fives -= 2) out[k++] = 25;
    for (; fives > 0; --fives) out[k++] = 5;
    for (; threes > 0; --threes) out[k++] = 3;
    for (; q16 > 0; --q16) out[k++] = 16;
    if (eight_four) {
        out[k++] = 8;
        out[k++] = 4;
    } else if (rem != 0) {
        out[k++] = rem == 3 ? 8 : (rem == 2 ? 4 : 2);
    }
    return k;
}

// An order as passes over shared memory: pass i runs the stage of radix a[i]
// and, where b[i] > 1, the stage of radix b[i] after it.
struct FxOrder {
    int count;
    int a[4], b[4];
    __host__ __device__ constexpr int radix(int i) const { return a[i] * b[i]; }
    // span of pass i's first stage
    __host__ __device__ constexpr int span(int i) const {
        int ns = 1;
        for (int j = 0; j < i; ++j) ns *= radix(j);
        return ns;
    }
    // twiddles of a stage of radix r over span ns (the first stage has none; an
    // even number per span offset)
    __host__ __device__ static constexpr int stage(int ns, int r) { return ns > 1 ? ns * ((r + 1) & ~1) : 0; }
    // twiddles ahead of pass i's
    __host__ __device__ constexpr int table(int i) const {
        int t = 0, ns = 1;
        for (int j = 0; j < i; ++j) {
            t += stage(ns, a[j]);
            if (b[j] > 1) t += stage(ns * a[j], b[j]);
            ns *= radix(j);
        }
        return t;
    }
    __host__ __device__ constexpr int table() const { return table(count); }
};

// The stages r[0 .. k) grouped into the fewest passes (at most four) of radix
// up to 25 whose last has a radix up to `last`; of those the grouping with the
// smallest largest radix.  count 0: none.
constexpr FxOrder fx_group(const int (&r)[16], int k, int last) {
    FxOrder best{};
    int best_top = 0;
    for (int cuts = 0; k > 0 && cuts < (1 << (k - 1)); ++cuts) {
        FxOrder o{};
        int top = 0, in_pass = 0;
        bool fits = true;
        for (int i = 0; i < k && fits; ++i) {
            if (i > 0 && ((cuts >> (i - 1)) & 1) == 0) {  // joins the stage before
                if (++in_pass > 2) fits = false;
                o.b[o.count - 1] = r[i];
            } else if (o.count == 4) {
                fits = false;
            } else {
                o.a[o.count] = r[i];
                o.b[o.count] = 1;
                in_pass = 1;
                ++o.count;
            }
            if (fits && o.radix(o.count - 1) > top) top = o.radix(o.count - 1);
        }
        if (!fits || top > 25 || o.radix(o.count - 1) > last || o.count < 2) continue;
        if (best.count == 0 || o.count < best.count || (o.count == best.count && top < best_top)) {
            best = o;
            best_top = top;
        }
    }
    return best;
}

// Row lengths 1250, 1280 and 2500 and column lengths 1600 and 3200 take their
// spectral chain's twiddles from the table of every w^r, not from w^1 by
// products as the runtime-planned transforms (and the luma-lock chain) do.
constexpr bool fx_table_twiddles(bool rows, int n) {
    return rows ? n == 1250 || n == 1280 || n == 2500 : n == 1600 || n == 3200;
}

// The FP16 form's order of a row plan (radices of ld_fxplans.h): four sequences
// (frame rows) choose the family; a row pass's last stage is taken in mirrored
// pairs of at most 16 values each.
constexpr FxOrder fx_row_order(int r1, int r2, int r3) {
    const int n = r1 * r2 * r3;
    int r[16] = {};
    const int k = plan_radices(n, 4 * n <= 12800, r);
    return fx_group(r, k, 16);
}
// ... and of a column plan: three sequences choose the family; the two plans of
// 1600 and of 3200 run their own radices.  None for 2500, 4800 and 5400, whose
// first two stages have the same radix of five or 25: the compiler contracts
// the second one's twiddle products otherwise there, and the bits differ.
constexpr FxOrder fx_col_order(int r1, int r2, int r3) {
    const int n = r1 * r2 * r3;
    if (fx_table_twiddles(false, n)) return FxOrder{3, {r1, r2, r3, 0}, {1, 1, 1, 0}};
    int r[16] = {};
    const int k = plan_radices(n, 3 * n <= 12800, r);
    if (k > 1 && r[0] == r[1] && r[0] % 5 == 0) return FxOrder{};
    return fx_group(r, k, 25);
}

}  // namespace ld
