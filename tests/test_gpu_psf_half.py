"""The compiled PSF sizes above 2048 with a pupil between a quarter and a half of
the size, whose transforms drop the zero half of the embedded pupil: the FP32
form's bank on them against the FP64 oracle.  (4096 would need a pupil above
1024, the largest there is.)"""
import pytest

from lensdiff_b200 import synthetic as S
from oracle import ld_oracle as O
from tests.helpers import PSF_TOL, rel_err
from tests.test_gpu_psf_plans import _sizes

LARGE = [n for n in _sizes() if 2048 < n < 4096]


def test_sizes_reach_the_largest_pupils_half():
    assert len(LARGE) >= 10


@pytest.mark.gpu
@pytest.mark.parametrize("size,pupil", [(n, 1024) for n in LARGE] + [(LARGE[0], LARGE[0] // 4 + 1)])
def test_half_zero_bank_matches_oracle(size, pupil):
    import torch

    from lensdiff_b200.backend import LensDiffPsfBankCache

    p = S.base_params(4000)
    p.apertureMode = 1
    p.bladeCount = 7
    p.roundness = 0.3
    p.centralObstruction = 0.2
    p.pupilResolution = pupil
    p.maxKernelRadiusPx = S.radius_percent(size // 4, 4000)
    p.phaseDefocus = 0.3
    p.spectralMode = 3
    p.wavelengthsNm = [560.0]
    p.rgbMode = 1
    np_, s, _ = O.resolve_sizes(p)
    assert (np_, s) == (pupil, size) and size < 4 * pupil and 2 * pupil <= size
    r0 = O.reference_first_zero(np_, s)
    p.diffractionScalePx = 100.0 * max(1.0, 2.0 * r0) / 4000
    ob = O.build_psf_bank(p, r0)
    cache = LensDiffPsfBankCache(0)
    _, kernels, st = cache.export_psf_bank(p, torch.cuda.current_stream())
    assert st.ok, st
    assert st.raw_psf_size == size
    for k, b in zip(kernels, ob.bins):
        assert k.shape == b.full.shape
        assert rel_err(k, b.full, b.full.max()) < PSF_TOL
    cache.close()
