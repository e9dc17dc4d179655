"""The blur at the edges of its tiles (64 pixels of a line per warp, four lines per block, 96 taps per
fill) and for every kind of pixel, against the oracle: equal to the last bit (src/d2bi.f90:1543-1624)."""
import numpy as np
import pytest

from oracle import stem_oracle as O
from simulated_tem_gb300 import imaging

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = imaging.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("nx,ny,t", [(1, 1, 1.0), (63, 3, 1.0), (64, 4, 2.0), (65, 5, 6.97), (96, 97, 3.3),
                                     (97, 1, 9.5), (1, 129, 9.6), (33, 160, 40.0), (40, 20, 0.1), (129, 66, 19.3)])
@pytest.mark.parametrize("kind", ["positive", "signed", "zeros", "wide", "special"])
def test_blur_equals_oracle(ctx, nx, ny, t, kind):
    rng = np.random.default_rng(nx * 1000 + ny)
    img = rng.random((nx, ny))
    if kind != "positive":
        img = img - 0.5
    if kind == "zeros":
        img[rng.random((nx, ny)) < 0.5] = 0.0
        img[rng.random((nx, ny)) < 0.2] = -0.0
    if kind == "wide":  # beyond the range of the integer products, subnormal numbers among them
        img = img * 2.0 ** rng.integers(-1070, 1000, (nx, ny))
    if kind == "special":
        img[nx // 2, ny // 2] = np.inf
        img[0, ny - 1] = np.nan
    with np.errstate(all="ignore"):
        want = O.gaussian_blur(img, t)
    assert np.array_equal(ctx.blur(img, t), want, equal_nan=True)
