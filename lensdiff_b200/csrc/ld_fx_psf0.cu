// ld_fx_psf0.cu — PSF passes of the plans LD_FX_PSF_0 (ld_fxplans.h).
#include "ld_fx_psf.cuh"
#include "ld_fxplans.h"

namespace ld {

bool fx_psf_0(int id, const PsfBankArgs& a, bool rows, cudaStream_t s) {
    switch (id) {
#define LD_FX_CASE(ID, A, B, C) \
    case ID: return psf_pass<Fx3<A, B, C>>(a, rows, s);
        LD_FX_PSF_0(LD_FX_CASE)
#undef LD_FX_CASE
        default: return false;
    }
}

}  // namespace ld
