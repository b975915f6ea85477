"""Kernels launched while the one before them drains: frames and lenses that
change without a host synchronisation in between give what synchronised ones
give, the caller's own kernels before and after included, launched directly and
replayed as graphs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from lensdiff_b200 import synthetic as S  # noqa: E402
from lensdiff_b200.backend import LensDiffPsfBankCache, image_request  # noqa: E402
from lensdiff_b200.types import LensDiffEnergyMode, LensDiffFftForm, LensDiffLookMode  # noqa: E402
from tests.test_gpu_modes import _field_lens, _lens  # noqa: E402

pytestmark = pytest.mark.gpu

# Two builds of one frame differ by the order of their FP64 ring sums and by the
# FP16 rounding that a last-bit difference moves; a frame or lens read too early
# differs by its contrast (here a factor 2 and 4 in brightness).
TOL = 1e-3
LENSES = {
    "plain": lambda: _lens(rgbMode=1, fftForm=LensDiffFftForm.OwnChosen),
    "split": lambda: _lens(rgbMode=1, lookMode=LensDiffLookMode.Split, coreGain=0.8, structureGain=1.2),
    "zones": lambda: _field_lens(rgbMode=1, energyMode=LensDiffEnergyMode.Preserve, fftForm=LensDiffFftForm.OwnChosen),
}


def _run(cache, lens, frames, stream, synchronised, cold):
    src, dst, out = torch.empty_like(frames[0]), torch.empty_like(frames[0]), []
    with torch.cuda.stream(stream):
        for i, f in enumerate(frames):
            src.copy_(f).mul_(2.0)  # the caller's kernels before ...
            p = lens.copy(phaseDefocus=0.1 * i) if cold else lens
            st = cache.render(image_request(src, dst, stream, frame_short_side=p.frameShortSidePx), p)
            assert st.ok, st
            out.append(dst * 1.0)  # ... and after
            if synchronised:
                torch.cuda.synchronize()
    torch.cuda.synchronize()
    assert cache.check_device_errors() == 0
    return out


@pytest.mark.parametrize("cold", [True, False])
@pytest.mark.parametrize("name", sorted(LENSES))
def test_unsynchronised_frames_match_synchronised_ones(name, cold):
    lens = LENSES[name]()
    base = torch.from_numpy(np.ascontiguousarray(S.make_frame(200, 120, 16, 1.0, 60.0, seed=5), np.float32)).cuda()
    frames = [base * (4.0 if i % 2 else 1.0) for i in range(6)]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    a, b = LensDiffPsfBankCache(0), LensDiffPsfBankCache(0)
    try:
        want = _run(a, lens, frames, stream, True, cold)
        got = _run(b, lens, frames, stream, False, cold)
        for w, g in zip(want, got):
            assert ((w - g).abs().max() / w.abs().max()).item() < TOL
    finally:
        a.close()
        b.close()
