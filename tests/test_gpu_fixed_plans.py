"""Every compiled column and row length, for the spectral, luma-lock and Mono
chains: a narrow (or low) frame whose grid takes exactly that length, against
the FP64 oracle, and against the runtime-planned transforms on the same grid
(to the FP32 rounding that separates two orders of one transform)."""
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


def _lengths(kind):
    text = "\n".join(re.findall(rf"#define LD_FX_{kind}_\d\(X\) \\\n((?:.*\\\n)*.*)", open(_PLANS).read()))
    return sorted({int(a) * int(b) * int(c) for a, b, c in re.findall(r"X\(\d+, (\d+), (\d+), (\d+)\)", text)})


# (chain, FFT form): three kernels, four (luma lock), one kernel and three
# drivers (Mono, always FP32)
CHAINS = [("spectral", 0), ("spectral", 1), ("luma", 0), ("luma", 1), ("mono", 0)]


def _cases(kind):
    # the Mono and luma-lock chains are compiled up to 3200 (kFxOtherMax)
    return [(n, c, f) for n in _lengths(kind) for c, f in CHAINS if c == "spectral" or n <= 3200]


def _lens(chain, form):
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
    p.fftForm = form
    if chain == "mono":
        p.spectralMode = 0
        p.wavelengthsNm = None
    elif chain == "luma":
        p.rgbMode = 0
        p.naturalMatrix = [[0.1, 0.2, 0.9], [0.1, 1.0, 0.2], [1.1, 0.1, 0.0]]
        p.styleMatrix = [[0.3, 0.4, 0.5], [0.2, 0.7, 0.3], [0.8, 0.2, 0.3]]
        p.spectrumForce = 0.5
    return p


def _matrices(p):
    if int(p.spectralMode) == 0:
        return None, None
    if int(p.rgbMode) == 0:
        return np.array(p.naturalMatrix), np.array(p.styleMatrix)
    m = O.gaussian_rgb_matrix(O.wavelengths(p), p.rgbGaussCenterNm, p.rgbGaussSigmaNm)
    return m, m


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
    assert len(_lengths("COLS")) >= 50 and all(n % 4 == 0 for n in _lengths("COLS"))
    assert len(_lengths("ROWS")) >= 45


# rows or columns of padding, until the grid's cost model takes the length
SPARE = (0, 16, 36, 46, 54, 80, 104, 120, 160, 190)


def _check(p, frame, out, grid):
    generic, grid2 = _render(p, frame, -1)
    assert grid2 == grid
    ref = O.render(frame, p, O.build_psf_bank(p), *_matrices(p))
    scale = float(ref[..., :3].max())
    assert np.abs(out - ref).max() / scale < OUT_TOL
    # (the luma lock divides FP16-rounded values: there the form's own rounding,
    # up to 3.5e-5 of the frame maximum on either side, is all that is compared)
    if int(p.rgbMode) != 0 or int(p.fftForm) == 0:
        assert np.abs(out - generic).max() / scale < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("n,chain,form", _cases("COLS"))
def test_column_length_matches_oracle(n, chain, form):
    p = _lens(chain, form)
    for spare in SPARE:
        frame = S.make_frame(64, n - 2 * R - spare, 200, 1.0, 50.0, seed=n)
        # the first and the last row carry highlights: both ends of the column
        frame[0, 3, :3] = 40.0
        frame[-1, 60, :3] = 30.0
        out, grid = _render(p, frame, 0)
        if grid[1] == n:
            break
    assert grid[1] == n
    _check(p, frame, out, grid)


@pytest.mark.gpu
@pytest.mark.parametrize("n,chain,form", _cases("ROWS"))
def test_row_length_matches_oracle(n, chain, form):
    p = _lens(chain, form)
    for spare in SPARE:
        # an odd width: the last pixel pair is half outside; 66 rows: a last
        # row tile that is partly padding
        frame = S.make_frame(2 * (n - R - spare) - 1, 66, 200, 1.0, 50.0, seed=n)
        frame[3, 0, :3] = 40.0
        frame[65, -1, :3] = 30.0
        out, grid = _render(p, frame, 0)
        if grid[0] == 2 * n:
            break
    assert grid[0] == 2 * n
    _check(p, frame, out, grid)
