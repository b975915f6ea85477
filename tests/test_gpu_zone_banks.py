"""Field zones whose canvas passes run several zones at a time, against the
same frame in the FP32 form, which builds each zone's bank by itself: groups of
all zones, of several with a remainder, and of one."""
import pytest

torch = pytest.importorskip("torch")

from lensdiff_b200 import synthetic as S  # noqa: E402
from lensdiff_b200.types import LensDiffEnergyMode, LensDiffFftForm, LensDiffLookMode  # noqa: E402
from tests.helpers import OUT_TOL, rel_err  # noqa: E402
from tests.test_gpu_modes import _field_lens, _render, cache  # noqa: E402,F401

pytestmark = pytest.mark.gpu


# 96 MB of canvases a group: 9 zones of 9 x 61^2 in one, 9 of 31 x 301^2 as
# 8 + 1, 4 of 31 x 601^2 as 2 + 2, 4 of 31 x 1025^2 one by one
@pytest.mark.parametrize("n,bins,radius", [(3, 9, 30), (3, 31, 150), (2, 31, 300), (2, 31, 512)])
@pytest.mark.parametrize("kw", [{}, {"lookMode": LensDiffLookMode.Split, "coreGain": 0.8, "structureGain": 1.2},
                                {"energyMode": LensDiffEnergyMode.Preserve, "anisotropyEmphasis": 0.0}])
def test_grouped_zone_banks_match_single_ones(cache, n, bins, radius, kw):
    p = _field_lens(fieldGrid=n, pupilResolution=128, maxKernelRadiusPx=S.radius_percent(radius, 160),
                    rgbMode=1,
                    wavelengthsNm=[400.0 + 300.0 * i / (bins - 1) for i in range(bins)], **kw)
    p = p.copy(frameShortSidePx=160)
    src = S.make_frame(240, 160, 30, 1.0, 120.0, seed=7)
    grouped = _render(cache, p.copy(fftForm=LensDiffFftForm.OwnChosen), src)
    single = _render(cache, p.copy(fftForm=LensDiffFftForm.OwnFp32), src)
    # each form is held to OUT_TOL of the oracle
    assert rel_err(grouped, single, single[..., :3].max()) < 2 * OUT_TOL
