// ld_fx_cols1.cu — column passes of the plans LD_FX_COLS_1 (ld_fxplans.h).
#include "ld_fx_cols.cuh"
#include "ld_fxplans.h"

namespace ld {

bool fx_cols_1(int id, const FrameArgs* fa, const KernelSpectraArgs* ka, cudaStream_t s) {
    switch (id) {
#define LD_FX_CASE(ID, A, B, C) \
    case ID: return cols_launch<Fx3<A, B, C>>(fa, ka, s);
        LD_FX_COLS_1(LD_FX_CASE)
#undef LD_FX_CASE
        default: return false;
    }
}

}  // namespace ld
