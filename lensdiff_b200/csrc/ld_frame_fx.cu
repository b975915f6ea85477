// ld_frame_fx.cu — the launchers of the fixed plans of ld_fxplans.h (their
// kernels are in ld_fx_rows*.cu, ld_fx_cols*.cu and ld_fx_psf*.cu) and the FP64 generation of
// the plans' stage twiddle tables.
//
// Each fx_launch_* returns false when no fixed instantiation covers the launch
// (another length, channel count or form); the caller then launches the
// runtime-planned kernel.
#include <cmath>
#include <vector>

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

// A row plan's inverse runs its radices in reverse: its tables follow.
std::vector<float2> fx_stage_table(int id) {
    std::vector<float2> out;
    const FxPlanDesc* d = fx_plan(id);
    if (d == nullptr) return out;
    append_stages({d->radix[0], d->radix[1], d->radix[2]}, &out);
    if (d->role == kFxRows) append_stages({d->radix[2], d->radix[1], d->radix[0]}, &out);
    return out;
}

}  // namespace ld
