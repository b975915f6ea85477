// ld_fx_rows4.cu — row passes of the plans LD_FX_ROWS_4 (ld_fxplans.h).
#include "ld_fx_rows.cuh"
#include "ld_fxplans.h"

namespace ld {

bool fx_rows_4(int id, int pass, const FrameArgs* fa, const KernelSpectraArgs* ka, int rows, cudaStream_t s) {
    switch (id) {
#define LD_FX_CASE(ID, A, B, C) \
    case ID: return rows_launch<FxRow<A, B, C>>(pass, fa, ka, rows, s);
        LD_FX_ROWS_4(LD_FX_CASE)
#undef LD_FX_CASE
        default: return false;
    }
}

}  // namespace ld
