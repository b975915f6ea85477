// ld_frame_fx.cu — the launchers of the fixed plans of ld_fxplans.h (their
// kernels are in ld_fx_rows*.cu, ld_fx_cols*.cu and ld_fx_psf*.cu) and the FP64 generation of
// the plans' stage twiddle tables.
//
// Each fx_launch_* returns false when no fixed instantiation covers the launch
// (another length, channel count or form); the caller then launches the
// runtime-planned kernel.
#include <cmath>
#include <vector>

#include "ld_fxorder.h"
#include "ld_fxplans.h"
#include "ld_internal.h"

namespace ld {
namespace {

bool cols_dispatch(int id, const FrameArgs* fa, const KernelSpectraArgs* ka, cudaStream_t s) {
    return fx_cols_0(id, fa, ka, s) || fx_cols_1(id, fa, ka, s) || fx_cols_2(id, fa, ka, s) ||
           fx_cols_3(id, fa, ka, s) || fx_cols_4(id, fa, ka, s) || fx_cols_5(id, fa, ka, s);
}

bool rows_dispatch(int id, int pass, const FrameArgs* fa, const KernelSpectraArgs* ka, int rows, cudaStream_t s) {
    return fx_rows_0(id, pass, fa, ka, rows, s) || fx_rows_1(id, pass, fa, ka, rows, s) ||
           fx_rows_2(id, pass, fa, ka, rows, s) || fx_rows_3(id, pass, fa, ka, rows, s) ||
           fx_rows_4(id, pass, fa, ka, rows, s) || fx_rows_5(id, pass, fa, ka, rows, s);
}

// The tables of the stages after the first of radices r[0], r[1], r[2]: for
// every such stage NS x RP entries w^(k r), w = exp(-2 pi i / (NS R)), k < NS,
// r < R (zero for r >= R), RP = R rounded up to even, as RP / 2 rows of NS
// pairs (w^(k 2q), w^(k (2q+1))): pair q of butterfly span k at q * NS + k, so
// the threads of a warp (consecutive k) read consecutive 16-byte pairs;
// evaluated in FP64.
void append_stages(const int (&radix)[3], std::vector<float2>* out) {
    int ns = 1;
    for (const int R : radix) {
        const int RP = (R + 1) & ~1;
        for (int q = 0; ns > 1 && q < RP / 2; ++q) {
            for (int k = 0; k < ns; ++k) {
                for (int r = 2 * q; r < 2 * q + 2; ++r) {
                    const double ang = -2.0 * M_PI * static_cast<double>(k) * r / static_cast<double>(ns * R);
                    out->push_back(r >= R ? make_float2(0.0f, 0.0f)
                                          : make_float2(static_cast<float>(std::cos(ang)), static_cast<float>(std::sin(ang))));
                }
            }
        }
        ns *= R;
    }
}

float2 root(long long k, long long n) {  // exp(-2 pi i k / n)
    const double a = -2.0 * M_PI * static_cast<double>(k) / static_cast<double>(n);
    return make_float2(static_cast<float>(std::cos(a)), static_cast<float>(std::sin(a)));
}

// The tables of the stages of `o` (ld_fxorder.h) in turn, in append_stages'
// layout, for a transform of length n.  products: w^r as the runtime-planned
// stage (fft_stage in ld_fft.cuh) forms it, w^(r-1) * w in FP32 from the
// length's table (a complex product there is two fused multiply-adds and two
// products); else every w^r from FP64.
void append_order(const FxOrder& o, int n, bool products, std::vector<float2>* out) {
    int ns = 1;
    for (int i = 0; i < o.count; ++i) {
        for (const int R : {o.a[i], o.b[i]}) {
            if (R == 1) continue;
            const int RP = (R + 1) & ~1;
            const size_t base = out->size();
            if (ns > 1) out->resize(base + static_cast<size_t>(ns) * RP, make_float2(0.0f, 0.0f));
            for (int k = 0; ns > 1 && k < ns; ++k) {
                const float2 w1 = root(static_cast<long long>(k) * (n / (ns * R)), n);
                float2 w = w1;
                for (int r = 0; r < R; ++r) {
                    float2 v = make_float2(1.0f, 0.0f);
                    if (r > 0 && products) {
                        v = w;
                        w = make_float2(std::fmaf(v.x, w1.x, -(v.y * w1.y)), std::fmaf(v.x, w1.y, v.y * w1.x));
                    } else if (r > 0) {
                        v = root(static_cast<long long>(k) * r, static_cast<long long>(ns) * R);
                    }
                    (*out)[base + (static_cast<size_t>(r / 2) * ns + k) * 2 + (r & 1)] = v;
                }
            }
            ns *= R;
        }
    }
}

}  // namespace

bool fx_launch_frame_rows(const FrameArgs& a, cudaStream_t s) {
    if (a.g.plan_m.fixed == 0) return false;
    return rows_dispatch(a.g.plan_m.fixed, kFxPassRows, &a, nullptr, 0, s);
}

bool fx_launch_frame_cols(const FrameArgs& a, cudaStream_t s) {
    if (a.g.plan_py.fixed == 0) return false;
    return cols_dispatch(a.g.plan_py.fixed, &a, nullptr, s);
}

bool fx_launch_frame_inverse(const FrameArgs& a, int rows, cudaStream_t s) {
    if (a.g.plan_m.fixed == 0) return false;
    return rows_dispatch(a.g.plan_m.fixed, kFxPassInverse, &a, nullptr, rows, s);
}

bool fx_launch_kspec_rows(const KernelSpectraArgs& a, cudaStream_t s) {
    if (a.g.plan_m.fixed == 0) return false;
    return rows_dispatch(a.g.plan_m.fixed, kFxPassKspecRows, nullptr, &a, 0, s);
}

bool fx_launch_kspec_cols(const KernelSpectraArgs& a, cudaStream_t s) {
    if (a.g.plan_py.fixed == 0) return false;
    return cols_dispatch(a.g.plan_py.fixed, nullptr, &a, s);
}

bool fx_launch_psf(const PsfBankArgs& a, bool rows, cudaStream_t s) {
    const int id = a.plan_s.fixed;
    if (id == 0 || a.want_energy) return false;
    return fx_psf_0(id, a, rows, s) || fx_psf_1(id, a, rows, s) || fx_psf_2(id, a, rows, s) || fx_psf_3(id, a, rows, s);
}

// A row plan's inverse runs its radices in reverse: its tables follow, then the
// FP16 form's order.
std::vector<float2> fx_stage_table(int id) {
    std::vector<float2> out;
    const FxPlanDesc* d = fx_plan(id);
    if (d == nullptr) return out;
    append_stages({d->radix[0], d->radix[1], d->radix[2]}, &out);
    if (d->role == kFxRows) append_stages({d->radix[2], d->radix[1], d->radix[0]}, &out);
    if (d->role != kFxPsf) {
        const bool rows = d->role == kFxRows;
        const FxOrder o = rows ? fx_row_order(d->radix[0], d->radix[1], d->radix[2])
                               : fx_col_order(d->radix[0], d->radix[1], d->radix[2]);
        append_order(o, d->n(), true, &out);
        if (fx_table_twiddles(rows, d->n())) append_order(o, d->n(), false, &out);
    }
    return out;
}

}  // namespace ld
