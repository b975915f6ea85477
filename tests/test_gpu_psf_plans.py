"""Every compiled PSF size: the FP32 form's bank on it against the FP64 oracle, for
a pupil of half the PSF (or the largest there is) and one below a quarter."""
import os
import re

import pytest

from lensdiff_b200 import synthetic as S
from oracle import ld_oracle as O
from tests.helpers import PSF_TOL, rel_err

_PLANS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lensdiff_b200", "csrc",
                      "ld_fxplans.h")


def _sizes():
    text = "\n".join(re.findall(r"#define LD_FX_PSF_\d\(X\) \\\n((?:.*\\\n)*.*)", open(_PLANS).read()))
    return sorted({int(a) * int(b) * int(c) for a, b, c in re.findall(r"X\(\d+, (\d+), (\d+), (\d+)\)", text)})


def test_psf_sizes_are_even():
    assert len(_sizes()) >= 30 and all(n % 2 == 0 for n in _sizes())


@pytest.mark.gpu
@pytest.mark.parametrize("half", [True, False])
@pytest.mark.parametrize("size", _sizes())
def test_bank_on_psf_size_matches_oracle(size, half):
    import torch

    from lensdiff_b200.backend import LensDiffPsfBankCache

    pupil = size // 2 if half else max(64, size // 4 - 5)
    if pupil > 1024:
        pytest.skip("pupils end at 1024")
    radius = size // 4
    if (half and size % 4 != 0) or max(2 * pupil, 512, 4 * radius) != size:
        pytest.skip("no kernel radius gives this size")
    p = S.base_params(4000)
    p.apertureMode = 1
    p.bladeCount = 7
    p.roundness = 0.3
    p.centralObstruction = 0.2
    p.pupilResolution = pupil
    # a small kernel canvas would shrink S = 4 R: half the sizes by the pupil alone
    p.maxKernelRadiusPx = S.radius_percent(40 if half else radius, 4000)
    p.phaseDefocus = 0.3
    p.spectralMode = 3
    p.wavelengthsNm = [420.0, 560.0, 690.0]
    p.rgbMode = 1
    np_, s, _ = O.resolve_sizes(p)
    if s != size:
        pytest.skip("no kernel radius gives this size")
    r0 = O.reference_first_zero(np_, s)
    p.diffractionScalePx = 100.0 * max(1.0, 2.0 * r0) / 4000  # footprints near half a window pixel
    ob = O.build_psf_bank(p, r0)
    cache = LensDiffPsfBankCache(0)
    _, kernels, st = cache.export_psf_bank(p, torch.cuda.current_stream())
    assert st.ok, st
    assert st.raw_psf_size == size
    for k, b in zip(kernels, ob.bins):
        assert k.shape == b.full.shape
        assert rel_err(k, b.full, b.full.max()) < PSF_TOL
    cache.close()
