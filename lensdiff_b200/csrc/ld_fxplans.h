// ld_fxplans.h — the transform lengths and radix orders compiled as fixed
// plans, shared by the host (planning, twiddle tables, the autotuner's
// candidate lists) and the kernels' translation units.
//
// Row plans (length M, half the grid's width) run on ld_fftx.cuh
// (ld_frame_fx.cu), column plans (length Py) on ld_fxpass.cuh (ld_fx_cols*.cu):
// every length from 300 to 5400 that the grid's cost model (choose_length in
// ld_host.cu) picks for three column sequences has one.  Where a length has
// several orders the autotuner times them on first use and keeps the fastest
// (the first is the default).  Odd radices lead where the length has them:
// their strided first-stage stores spread over the shared-memory banks.
#pragma once

namespace ld {

enum { kFxRows = 1, kFxCols = 2 };

struct FxPlanDesc {
    int id;         // 0 means "no fixed plan"
    int role;       // kFxRows, kFxCols
    int count;      // stages
    int radix[3];   // radix of each stage, first stage first
    constexpr int n() const { return radix[0] * radix[1] * (count > 2 ? radix[2] : 1); }
};

// Column plans X(id, R1, R2, R3), in the groups that the translation units
// ld_fx_cols0.cu .. ld_fx_cols5.cu compile.
#define LD_FX_COLS_0(X) \
    X(20, 5, 5, 12) X(26, 5, 10, 10) X(32, 9, 8, 10) X(38, 25, 5, 8) X(44, 9, 9, 16) \
    X(50, 15, 10, 12) X(56, 25, 10, 10) X(62, 25, 8, 16) X(68, 12, 16, 24)
#define LD_FX_COLS_1(X) \
    X(21, 5, 8, 8) X(27, 8, 8, 8) X(33, 3, 16, 16) X(39, 8, 8, 16) X(45, 9, 10, 16) \
    X(51, 15, 8, 16) X(57, 20, 8, 16) X(63, 9, 24, 16) X(69, 25, 12, 16)
#define LD_FX_COLS_2(X) \
    X(22, 3, 8, 16) X(28, 9, 8, 8) X(34, 5, 10, 16) X(40, 9, 10, 12) X(46, 15, 10, 10) \
    X(52, 25, 8, 10) X(58, 15, 12, 15) X(64, 15, 15, 16) X(70, 20, 16, 16)
#define LD_FX_COLS_3(X) \
    X(23, 5, 8, 10) X(29, 5, 10, 12) X(35, 9, 8, 12) X(41, 9, 8, 16) X(47, 25, 16, 4) \
    X(53, 8, 16, 16) X(59, 15, 12, 16) X(65, 15, 16, 16) X(71, 9, 24, 24)
#define LD_FX_COLS_4(X) \
    X(24, 9, 12, 4) X(30, 5, 8, 16) X(36, 9, 10, 10) X(42, 15, 8, 10) X(48, 25, 4, 16) \
    X(54, 15, 9, 16) X(60, 25, 8, 15) X(66, 16, 16, 16) X(72, 15, 15, 24)
#define LD_FX_COLS_5(X) \
    X(25, 5, 8, 12) X(31, 9, 8, 9) X(37, 15, 8, 8) X(43, 5, 16, 16) X(49, 9, 12, 16) \
    X(55, 9, 16, 16) X(61, 25, 16, 8) X(67, 15, 12, 24)
#define LD_FX_COL_DESC(ID, A, B, C) {ID, kFxCols, 3, {A, B, C}},
constexpr FxPlanDesc kFxPlans[] = {
    {1, kFxRows, 3, {25, 25, 4}},
    {2, kFxRows, 3, {25, 4, 25}},
    {5, kFxRows, 3, {25, 25, 2}},
    {6, kFxRows, 3, {25, 2, 25}},
    {9, kFxRows, 3, {5, 16, 16}},
    {10, kFxRows, 3, {16, 5, 16}},
    LD_FX_COLS_0(LD_FX_COL_DESC) LD_FX_COLS_1(LD_FX_COL_DESC) LD_FX_COLS_2(LD_FX_COL_DESC)
    LD_FX_COLS_3(LD_FX_COL_DESC) LD_FX_COLS_4(LD_FX_COL_DESC) LD_FX_COLS_5(LD_FX_COL_DESC)
};
#undef LD_FX_COL_DESC

inline const FxPlanDesc* fx_plan(int id) {
    for (const FxPlanDesc& d : kFxPlans)
        if (d.id == id) return &d;
    return nullptr;
}

// Fixed plans of length n for `role`, in preference order; returns how many (<= max).
inline int fx_candidates(int n, int role, int* ids, int max) {
    int k = 0;
    for (const FxPlanDesc& d : kFxPlans)
        if (k < max && d.role == role && d.n() == n) ids[k++] = d.id;
    return k;
}

}  // namespace ld
