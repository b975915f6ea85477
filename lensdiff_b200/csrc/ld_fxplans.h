// ld_fxplans.h — the transform lengths and radix orders compiled as fixed
// plans, shared by the host (planning, twiddle tables) and the kernels'
// translation units.
//
// Row plans (length M, half the grid's width: ld_fx_rows*.cu) and column plans
// (length Py: ld_fx_cols*.cu) run on ld_fxpass.cuh.  Every length that the
// grid's cost model (choose_length in ld_host.cu) picks for the spectral
// chains has one: columns from 300 to 5400, rows from 256 to 4096.  Column
// lengths 1600 and 3200 have two orders: frames that composite directly run the
// second from a context's second such frame on (the kernel spectra that the
// first one built stay as they are), others the first.  (They are within 3 % of
// one another; an order that changes moves the FP16 form's results by up to
// 2e-5, so each frame keeps the one it has always had.)  Odd radices lead where the length has them: their
// strided first-stage stores spread over the shared-memory banks.  A row plan's last radix is also its inverse's first, and is taken in
// pairs of mirrored butterflies: a small one.  PSF plans (length S:
// ld_fx_psf*.cu) cover the common PSF sizes; their first radix is a multiple
// of four, whose transforms drop the zero half of the embedded pupil.
#pragma once

namespace ld {

enum { kFxRows = 1, kFxCols = 2, kFxPsf = 3 };

struct FxPlanDesc {
    int id;         // 1 .. 255 (0 means "no fixed plan")
    int role;       // kFxRows, kFxCols, kFxPsf
    int radix[3];   // radix of each stage, first stage first
    constexpr int n() const { return radix[0] * radix[1] * radix[2]; }
};

// Column plans X(id, R1, R2, R3), in the groups that the translation units
// ld_fx_cols0.cu .. ld_fx_cols5.cu compile.
#define LD_FX_COLS_0(X) \
    X(20, 5, 5, 12) X(26, 5, 10, 10) X(32, 9, 8, 10) X(38, 25, 5, 8) X(44, 9, 9, 16) \
    X(50, 15, 10, 12) X(56, 25, 10, 10) X(62, 25, 16, 8) X(68, 12, 16, 24)
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
    X(55, 9, 16, 16) X(61, 25, 8, 16) X(67, 15, 12, 24)
// Row plans X(id, R1, R2, R3), in the groups of ld_fx_rows0.cu .. ld_fx_rows5.cu.
#define LD_FX_ROWS_0(X) \
    X(100, 8, 8, 4) X(106, 5, 10, 9) X(112, 5, 16, 8) X(118, 9, 10, 10) X(124, 25, 10, 5) \
    X(130, 25, 8, 8) X(136, 15, 16, 9) X(142, 25, 12, 10) X(148, 16, 16, 16)
#define LD_FX_ROWS_1(X) \
    X(101, 5, 12, 5) X(107, 5, 10, 10) X(113, 15, 9, 5) X(119, 15, 8, 8) X(125, 10, 16, 8) \
    X(131, 9, 16, 12) X(137, 12, 16, 12) X(143, 25, 25, 5)
#define LD_FX_ROWS_2(X) \
    X(102, 5, 8, 8) X(108, 8, 8, 8) X(114, 9, 10, 8) X(120, 25, 5, 8) X(126, 9, 16, 9) \
    X(132, 15, 12, 10) X(138, 25, 10, 10) X(144, 25, 16, 8)
#define LD_FX_ROWS_3(X) \
    X(103, 5, 15, 5) X(109, 9, 8, 8) X(115, 12, 8, 8) X(121, 16, 8, 8) X(127, 15, 9, 10) \
    X(133, 25, 15, 5) X(139, 20, 16, 8) X(145, 24, 16, 9)
#define LD_FX_ROWS_4(X) \
    X(104, 5, 10, 8) X(110, 5, 12, 10) X(116, 5, 16, 10) X(122, 15, 15, 5) X(128, 15, 12, 8) \
    X(134, 25, 10, 8) X(140, 15, 15, 12) X(146, 25, 16, 9)
#define LD_FX_ROWS_5(X) \
    X(105, 9, 12, 4) X(111, 5, 25, 5) X(117, 9, 12, 8) X(123, 15, 10, 8) X(129, 15, 10, 10) \
    X(135, 16, 16, 8) X(141, 15, 16, 12) X(147, 20, 16, 12)

// PSF plans X(id, R1, R2, R3), in the groups of ld_fx_psf0.cu .. ld_fx_psf3.cu.
#define LD_FX_PSF_0(X) \
    X(160, 8, 8, 8) X(164, 8, 9, 9) X(168, 12, 9, 8) X(172, 16, 8, 8) X(176, 16, 10, 8) \
    X(180, 16, 12, 8) X(184, 16, 12, 10) X(188, 16, 16, 9) X(192, 20, 15, 10) X(196, 16, 16, 15)
#define LD_FX_PSF_1(X) \
    X(161, 8, 9, 8) X(165, 16, 9, 5) X(169, 20, 9, 5) X(173, 12, 10, 9) X(177, 16, 9, 9) \
    X(181, 16, 10, 10) X(185, 20, 10, 10) X(189, 16, 15, 10) X(193, 16, 16, 12) X(197, 20, 20, 10)
#define LD_FX_PSF_2(X) \
    X(162, 12, 10, 5) X(166, 12, 8, 8) X(170, 12, 10, 8) X(174, 16, 9, 8) X(178, 16, 10, 9) \
    X(182, 16, 12, 9) X(186, 16, 16, 8) X(190, 16, 16, 10) X(194, 20, 16, 10) X(198, 16, 16, 16)
#define LD_FX_PSF_3(X) \
    X(163, 16, 8, 5) X(167, 16, 10, 5) X(171, 20, 10, 5) X(175, 12, 10, 10) X(179, 20, 15, 5) \
    X(183, 20, 10, 9) X(187, 16, 15, 9) X(191, 16, 15, 12) X(195, 20, 15, 12)

#define LD_FX_COL_DESC(ID, A, B, C) {ID, kFxCols, {A, B, C}},
#define LD_FX_ROW_DESC(ID, A, B, C) {ID, kFxRows, {A, B, C}},
#define LD_FX_PSF_DESC(ID, A, B, C) {ID, kFxPsf, {A, B, C}},
constexpr FxPlanDesc kFxPlans[] = {
    LD_FX_COLS_0(LD_FX_COL_DESC) LD_FX_COLS_1(LD_FX_COL_DESC) LD_FX_COLS_2(LD_FX_COL_DESC)
    LD_FX_COLS_3(LD_FX_COL_DESC) LD_FX_COLS_4(LD_FX_COL_DESC) LD_FX_COLS_5(LD_FX_COL_DESC)
    LD_FX_ROWS_0(LD_FX_ROW_DESC) LD_FX_ROWS_1(LD_FX_ROW_DESC) LD_FX_ROWS_2(LD_FX_ROW_DESC)
    LD_FX_ROWS_3(LD_FX_ROW_DESC) LD_FX_ROWS_4(LD_FX_ROW_DESC) LD_FX_ROWS_5(LD_FX_ROW_DESC)
    LD_FX_PSF_0(LD_FX_PSF_DESC) LD_FX_PSF_1(LD_FX_PSF_DESC) LD_FX_PSF_2(LD_FX_PSF_DESC) LD_FX_PSF_3(LD_FX_PSF_DESC)
};
#undef LD_FX_COL_DESC
#undef LD_FX_ROW_DESC
#undef LD_FX_PSF_DESC

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
