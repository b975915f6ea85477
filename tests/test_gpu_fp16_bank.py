"""A bank with a box filter in the FP16 form keeps its FP32 bits, which its
half-rounded kernel spectra amplify: a log-encoded frame through a lens much
finer than a pixel against the frame that the form has always given (its error
against the FP64 oracle is about 6e-4 and says nothing about the bits).  Another
order of the rescale's sums moves it by 5e-5 to 7e-5 of its norm."""
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from lensdiff_b200 import synthetic as S  # noqa: E402
from lensdiff_b200.backend import LensDiffPsfBankCache, image_request  # noqa: E402

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "fp16_filtered_bank.npz")
WIDTH, HEIGHT = 160, 96
# FP32 outputs that are the same to rounding lie within 2e-5 of each other
SAME = 2e-5


def _davinci(x):
    log = (np.log2(np.maximum(x, 0.0) + 0.0075) + 7.0) * 0.07329248
    return np.where(x <= 0.00262409, x * 10.44426855, log)


def _inputs(seed):
    rng = np.random.default_rng(seed)
    frame = np.zeros((HEIGHT, WIDTH, 4), np.float64)
    frame[..., :3] = np.linspace(0.0, 0.2, WIDTH)[None, :, None] + 0.05
    ys, xs = rng.integers(0, HEIGHT, 24), rng.integers(0, WIDTH, 24)
    frame[ys, xs, :3] = np.exp(rng.uniform(0.0, np.log(1000.0), 24))[:, None] * np.array([1.0, 0.9, 0.8])
    frame[..., :3] = _davinci(frame[..., :3])
    frame[..., 3] = 1.0
    p = S.base_params(HEIGHT)
    p.apertureMode = 1
    p.bladeCount = 6
    p.roundness = 0.4
    p.pupilResolution = 333
    p.maxKernelRadiusPx = S.radius_percent(20, HEIGHT)
    p.diffractionScalePx = 1.0
    p.phaseDefocus = 0.25
    p.phaseSpherical = 0.1
    p.noll = [0.0, 0.0] + [float(v) for v in rng.normal(0.0, 0.09, 14)] + [0.0] * 7
    p.spectralMode = 3
    p.wavelengthsNm = [400.0, 550.0, 700.0]
    p.rgbMode = 1
    p.inputTransfer = 1
    p.fftForm = 1
    return p, frame.astype(np.float32)


def _render(p, frame, mode):
    cache = LensDiffPsfBankCache(0)
    cache.set_autotune(mode)
    stream = torch.cuda.Stream()
    src = torch.from_numpy(frame).cuda()
    dst = torch.zeros_like(src)
    torch.cuda.synchronize()
    st = cache.render(image_request(src, dst, stream, frame_short_side=HEIGHT), p)
    stream.synchronize()
    assert st.ok, st
    assert cache.check_device_errors() == 0
    cache.close()
    return dst.cpu().numpy()[..., :3]


SEEDS = (1, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [-1, 0, 1])
@pytest.mark.parametrize("seed", SEEDS)
def test_filtered_bank_keeps_its_bits(seed, mode):
    p, frame = _inputs(seed)
    want = np.load(GOLDEN)[f"seed{seed}"].astype(np.float64)
    got = _render(p, frame, mode)
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < SAME
