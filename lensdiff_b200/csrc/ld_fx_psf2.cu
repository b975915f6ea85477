// ld_fx_psf2.cu — PSF passes of the plans LD_FX_PSF_2 (ld_fxplans.h).
#include "ld_fx_psf.cuh"
#include "ld_fxplans.h"

namespace ld {

bool fx_psf_2(int id, const PsfBankArgs& a, bool rows, cudaStream_t s) {
    switch (id) {
#define LD_FX_CASE(ID, A, B, C) \
    case ID: return psf_pass<Fx3<A, B, C>>(a, rows, s);
        LD_FX_PSF_2(LD_FX_CASE)
#undef LD_FX_CASE
        default: return false;
    }
}

}  // namespace ld
