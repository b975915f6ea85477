"""The FP16 form's stored halves do not depend on which kernels made them: for
every compiled column and row length, the passes that store half (or feed a
store of half) run the stages of the runtime-planned transforms with the same
arithmetic, so a frame through them equals the same frame through the
runtime-planned ones.  Another order of the stages moves about one stored half
in a hundred, which shows here as 3e-7 to 3e-6 of the norm (and as up to 5e-5 in
small log-encoded frames)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from lensdiff_b200 import synthetic as S  # noqa: E402
from tests.test_gpu_fixed_plans import R, SPARE, _lengths, _lens, _render  # noqa: E402

pytestmark = pytest.mark.gpu

# Lengths whose spectral chain takes its twiddles from the full table
# (fx_table_twiddles in ld_fxorder.h): the runtime-planned transforms form them
# by products, so there the two are different computations.
TABLE_COLS, TABLE_ROWS = (1600, 3200), (1250, 1280, 2500)
# The rows' inverse transforms follow the last store of half and differ in
# order: 2^-24 sqrt(log2 n) <= 2.2e-7 of the effect's norm, which is less than
# half of these frames'.
INVERSE = 1e-7


def _unfiltered(chain):
    # samples less than one PSF pixel apart: the bank's sums then have one
    # order, and two contexts build the same bank to the bit
    p = _lens(chain, 1)
    p.diffractionScalePx = 60.0
    return p


@pytest.mark.parametrize("n,chain", [(n, c) for n in _lengths("COLS") for c in ("spectral", "luma")
                                     if (c == "spectral" or n <= 3200) and not (c == "spectral" and n in TABLE_COLS)])
def test_column_length_keeps_the_bits(n, chain):
    p = _unfiltered(chain)
    for spare in SPARE:
        frame = S.make_frame(64, n - 2 * R - spare, 200, 1.0, 50.0, seed=n)
        out, grid = _render(p, frame, 0)
        if grid[1] == n:
            break
    assert tuple(grid) == (96, n)  # rows of 48: runtime-planned in both
    assert np.array_equal(out, _render(p, frame, -1)[0])


@pytest.mark.parametrize("n", [n for n in _lengths("ROWS") if n not in TABLE_ROWS])
def test_row_length_keeps_the_bits(n):
    p = _unfiltered("spectral")
    for spare in SPARE:
        frame = S.make_frame(2 * (n - R - spare) - 1, 66, 200, 1.0, 50.0, seed=n)
        out, grid = _render(p, frame, 0)
        if grid[0] == 2 * n:
            break
    assert grid[0] == 2 * n
    generic = _render(p, frame, -1)[0].astype(np.float64)
    assert np.linalg.norm(out - generic) / np.linalg.norm(generic) < INVERSE
