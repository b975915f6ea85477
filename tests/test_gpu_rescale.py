"""The lambda-rescale against the FP64 oracle: box-filtered at footprints from
just above one window pixel to the clamped maximum, unfiltered up to one
window pixel per canvas pixel, and banks with both kinds of wavelength."""
import pytest

from lensdiff_b200 import synthetic as S
from oracle import ld_oracle as O
from tests.helpers import PSF_TOL, rel_err

pytestmark = pytest.mark.gpu


# (pupil, kernel radius, footprint at 550 nm): a run of 2 pixels, the 6-tap
# edge from both sides, taps more than a pixel apart, and the clamp at 20;
# canvases of one ragged tile and of several; then footprints of one window
# pixel and below: both kinds in one bank (1.02 and 0.99 at 400-700 nm), and
# the unfiltered kernel's tiles of 16, 64 and 128 rows with radii on and next
# to multiples of the tile sides
@pytest.mark.parametrize("pupil,radius,footprint", [
    (128, 5, 1.02), (128, 29, 2.5), (128, 40, 5.9), (128, 33, 6.1), (256, 100, 11.0), (256, 20, 60.0),
    (128, 64, 0.99), (128, 4, 0.7), (128, 31, 0.6), (128, 32, 0.3), (128, 260, 0.7), (128, 255, 0.35),
])
@pytest.mark.parametrize("emphasis", [0.0, 0.3])
def test_rescaled_bank_matches_oracle(pupil, radius, footprint, emphasis):
    import torch

    from lensdiff_b200.backend import LensDiffPsfBankCache

    p = S.base_params(200)
    p.apertureMode = 1
    p.bladeCount = 6
    p.roundness = 0.2
    p.pupilResolution = pupil
    p.maxKernelRadiusPx = S.radius_percent(radius, 200)
    p.phaseDefocus = 0.2
    p.anisotropyEmphasis = emphasis
    p.spectralMode = 3
    p.wavelengthsNm = [400.0, 550.0, 700.0] if radius < 200 else [400.0 + 20.0 * i for i in range(16)]
    p.rgbMode = 1
    np_, size, _ = O.resolve_sizes(p)
    r0 = O.reference_first_zero(np_, size)
    p.diffractionScalePx = 100.0 * (r0 / footprint) / 200
    ob = O.build_psf_bank(p, r0)
    cache = LensDiffPsfBankCache(0)
    _, kernels, st = cache.export_psf_bank(p, torch.cuda.current_stream())
    assert st.ok, st
    for k, b in zip(kernels, ob.bins):
        assert k.shape == b.full.shape
        assert rel_err(k, b.full, b.full.max()) < PSF_TOL
    cache.close()
