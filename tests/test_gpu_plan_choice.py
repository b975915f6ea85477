"""Which compiled radix order a frame runs on is settled without the GPU: the
first composite frame of a grid does not wait for it, every context takes the
same ones, and a length that is both a row and a column length of a grid
answers for the role that has several."""
import pytest

torch = pytest.importorskip("torch")

from lensdiff_b200 import synthetic as S  # noqa: E402
from lensdiff_b200.backend import LensDiffPsfBankCache, image_request  # noqa: E402

pytestmark = pytest.mark.gpu
R = 16


def _lens(preserve=False):
    p = S.base_params(64)
    p.pupilResolution = 64
    p.maxKernelRadiusPx = S.radius_percent(R, 64)
    p.diffractionScalePx = 60.0
    p.spectralMode = 3
    p.wavelengthsNm = [450.0, 550.0, 640.0]
    p.rgbMode = 1
    p.fftForm = 1
    if preserve:
        p.energyMode = 0
    return p


def _request(width, height, stream):
    src = torch.from_numpy(S.make_frame(width, height, 200, 1.0, 50.0, seed=5)).cuda()
    dst = torch.zeros_like(src)
    torch.cuda.synchronize()
    return image_request(src, dst, stream, frame_short_side=64)


def _choices(n, contexts):
    out = []
    for _ in range(contexts):
        cache = LensDiffPsfBankCache(0)
        stream = torch.cuda.Stream()
        st = cache.render(_request(2 * n - 2 * R - 32, n - 2 * R, stream), _lens())
        assert st.ok, st
        assert st.grid_used == (2 * n, n)
        c = cache.autotune_choice(n)
        assert c is not None and c[2] > 0.0
        out.append(c[0])
        cache.close()
    return out


@pytest.mark.parametrize("n,orders", [(1600, [(25, 16, 4), (25, 4, 16)]), (3200, [(25, 16, 8), (25, 8, 16)])])
def test_column_orders_are_reported_and_settled(n, orders):
    got = _choices(n, 3)
    assert got[0] in orders
    assert got == got[:1] * 3


def test_first_composite_frame_does_not_wait():
    cache = LensDiffPsfBankCache(0)
    stream = torch.cuda.Stream()
    rq = _request(64, 540, stream)
    # buffers, kernels and calibration of the grid, by a frame that does not composite directly
    for _ in range(2):
        assert cache.render(rq, _lens(preserve=True)).ok
    stream.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(400_000_000)  # 0.2 s
        done = torch.cuda.Event()
        done.record(stream)
    st = cache.render(rq, _lens())
    waited = done.query()
    stream.synchronize()
    assert st.ok, st
    assert not waited
    cache.close()


@pytest.mark.parametrize("n", [1600, 3200])
def test_orders_of_a_contexts_frames(n):
    """A context's first directly composited frame runs the first column order and
    its kernel spectra stay on it; later frames, and kernel spectra of new lenses,
    run the last.  Shown to the bit against the orders pinned one by one (the
    lens has no box filter, so two contexts build the same bank)."""
    stream = torch.cuda.Stream()
    rq = _request(64, n - 2 * R, stream)
    new = _lens().copy(phaseDefocus=0.3)

    def frames(steps):
        cache, out = LensDiffPsfBankCache(0), []
        for mode, lens in steps:
            cache.set_autotune(mode)
            st = cache.render(rq, lens)
            stream.synchronize()
            assert st.ok and st.grid_used[1] == n, st
            out.append(rq.dst.data.cpu().numpy())
        cache.close()
        return out

    first, warm, cold = frames([(1, _lens()), (1, _lens()), (1, new)])
    want_first, want_warm = frames([(2, _lens()), (3, _lens())])
    want_cold, = frames([(3, new)])
    assert (first == want_first).all()
    assert (warm == want_warm).all()
    assert (cold == want_cold).all()
    assert not (want_first == want_warm).all()  # the orders do differ
