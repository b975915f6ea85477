"""A memory budget that holds a frame with field zones when one zone's canvases
are held at a time holds it: the canvases of several zones together are not
taken from it."""
import pytest

torch = pytest.importorskip("torch")

from lensdiff_b200 import synthetic as S  # noqa: E402
from lensdiff_b200.backend import LensDiffPsfBankCache, image_request  # noqa: E402
from lensdiff_b200.types import LensDiffFftForm  # noqa: E402
from tests.helpers import rel_err  # noqa: E402
from tests.test_gpu_modes import _field_lens  # noqa: E402

pytestmark = pytest.mark.gpu


# What the frame needs with one zone's canvases, and 1 MB for tables: eight
# zones' canvases of the first lens are 79 MB more, two zones' of the second 45.
@pytest.mark.parametrize("n,bins,radius,megabytes", [(3, 31, 150, 659.9), (2, 31, 300, 974.0)])
def test_zones_render_within_one_zones_canvases(n, bins, radius, megabytes):
    p = _field_lens(fieldGrid=n, pupilResolution=128, maxKernelRadiusPx=S.radius_percent(radius, 160), rgbMode=1,
                    wavelengthsNm=[400.0 + 300.0 * i / (bins - 1) for i in range(bins)])
    p = p.copy(frameShortSidePx=160, fftForm=LensDiffFftForm.OwnChosen)
    src = torch.from_numpy(S.make_frame(240, 160, 30, 1.0, 120.0, seed=7)).cuda()
    out = []
    for budget in (0, int(megabytes * 1e6)):
        cache = LensDiffPsfBankCache(0, hbm_budget_bytes=budget)
        stream, dst = torch.cuda.Stream(), torch.zeros_like(src)
        torch.cuda.synchronize()
        st = cache.render(image_request(src, dst, stream, frame_short_side=160), p)
        stream.synchronize()
        assert st.ok, st
        out.append(dst.cpu().numpy())
        cache.close()
    # the same kernels over groups of other sizes: FP64 sums in another order,
    # whose rounding to float may move the FP16 form's stored halves
    assert rel_err(out[1], out[0], out[0][..., :3].max()) < 1e-5
