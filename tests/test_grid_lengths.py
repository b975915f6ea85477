"""Every frame height up to the largest transform has a grid: also those just
above a length that the transforms have, where the next multiple of four among
them is more than a tenth longer (649-654 and 1297-1309 rows with the kernel's
reach)."""
import numpy as np
import pytest

from lensdiff_b200 import abi
from lensdiff_b200 import synthetic as S
from oracle import ld_oracle as O
from tests.helpers import OUT_TOL

R = 16


def _lens(form):
    p = S.base_params(64)
    p.pupilResolution = 64
    p.maxKernelRadiusPx = S.radius_percent(R, 64)
    p.diffractionScalePx = 5.0
    p.phaseDefocus = 0.2
    p.spectralMode = 3
    p.wavelengthsNm = [450.0, 550.0, 640.0]
    p.rgbMode = 1
    p.fftForm = form
    return p


def test_every_height_has_a_grid():
    lib, p = abi.lib(), abi.to_abi_params(_lens(0))
    longest = 5400  # three interleaved columns of 16384 values
    refused = [rows for rows in range(2 * R + 1, longest + 1) if lib.ld_estimate_device_bytes(p, 64, rows - 2 * R) == 0]
    assert refused == []
    assert lib.ld_estimate_device_bytes(p, 64, longest + 1 - 2 * R) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("rows,grid", [(649, 720), (654, 720), (1297, 1440), (1309, 1440)])
def test_rows_between_grids_match_oracle(rows, grid, form):
    import torch

    from lensdiff_b200.backend import LensDiffPsfBankCache, image_request

    p = _lens(form)
    frame = S.make_frame(64, rows - 2 * R, 200, 1.0, 50.0, seed=rows)
    frame[0, 3, :3] = 40.0
    frame[-1, 60, :3] = 30.0
    cache = LensDiffPsfBankCache(0)
    stream = torch.cuda.Stream()
    src = torch.from_numpy(frame).cuda()
    dst = torch.full_like(src, -7.0)
    torch.cuda.synchronize()
    st = cache.render(image_request(src, dst, stream, frame_short_side=64), p)
    stream.synchronize()
    assert st.ok, st
    assert st.grid_used[1] == grid
    assert cache.check_device_errors() == 0
    m = O.gaussian_rgb_matrix(O.wavelengths(p), p.rgbGaussCenterNm, p.rgbGaussSigmaNm)
    ref = O.render(frame, p, O.build_psf_bank(p), m, m)
    assert np.abs(dst.cpu().numpy() - ref).max() / float(ref[..., :3].max()) < OUT_TOL
    cache.close()
