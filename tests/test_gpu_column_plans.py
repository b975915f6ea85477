"""Every compiled column length: a narrow frame whose grid takes exactly that
length, against the FP64 oracle, and against the runtime-planned transforms
on the same grid (to the FP32 rounding that separates two orders of one
transform)."""
import os
import re

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from lensdiff_b200 import synthetic as S  # noqa: E402
from lensdiff_b200.backend import LensDiffPsfBankCache, image_request  # noqa: E402
from oracle import ld_oracle as O  # noqa: E402
from tests.helpers import OUT_TOL  # noqa: E402

_PLANS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lensdiff_b200", "csrc",
                      "ld_fxplans.h")
R = 16


def _lengths():
    text = open(_PLANS).read()
    text = text[text.index("#define LD_FX_COLS_0"):text.index("LD_FX_COL_DESC")]
    return sorted({int(a) * int(b) * int(c) for a, b, c in re.findall(r"X\(\d+, (\d+), (\d+), (\d+)\)", text)})


def _lens():
    p = S.base_params(64)
    p.apertureMode = 1
    p.bladeCount = 5
    p.pupilResolution = 64
    p.maxKernelRadiusPx = S.radius_percent(R, 64)
    p.diffractionScalePx = 5.0
    p.phaseDefocus = 0.2
    p.spectralMode = 3
    p.wavelengthsNm = [450.0, 550.0, 640.0]
    p.rgbMode = 1
    return p


def _render(p, frame, mode):
    cache = LensDiffPsfBankCache(0)
    cache.set_autotune(mode)
    stream = torch.cuda.Stream()
    src = torch.from_numpy(frame).cuda()
    dst = torch.full_like(src, -7.0)
    torch.cuda.synchronize()
    st = cache.render(image_request(src, dst, stream, frame_short_side=64), p)
    stream.synchronize()
    assert st.ok, st
    assert cache.check_device_errors() == 0
    cache.close()
    return dst.cpu().numpy(), st.grid_used


def test_column_lengths_are_multiples_of_four():
    lengths = _lengths()
    assert len(lengths) >= 50 and all(n % 4 == 0 for n in lengths)


@pytest.mark.gpu
@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("n", _lengths())
def test_column_length_matches_oracle(n, form):
    p = _lens().copy(fftForm=form)
    for spare in (0, 46, 54, 104, 160, 190):  # rows of padding, until the grid's cost model takes this length
        frame = S.make_frame(64, n - 2 * R - spare, 200, 1.0, 50.0, seed=n)
        # the first and the last row carry highlights: both ends of the column
        frame[0, 3, :3] = 40.0
        frame[-1, 60, :3] = 30.0
        out, grid = _render(p, frame, 0)
        if grid[1] == n:
            break
    assert grid[1] == n
    generic, grid2 = _render(p, frame, -1)
    assert grid2 == grid
    m = O.gaussian_rgb_matrix(O.wavelengths(p), p.rgbGaussCenterNm, p.rgbGaussSigmaNm)
    ref = O.render(frame, p, O.build_psf_bank(p), m, m)
    scale = float(ref[..., :3].max())
    assert np.abs(out - ref).max() / scale < OUT_TOL
    assert np.abs(out - generic).max() / scale < 1e-5
