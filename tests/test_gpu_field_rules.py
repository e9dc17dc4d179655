"""The rules that choose between two ways of computing a field or an integration, on both sides of each."""
import numpy as np
import pytest

from simulated_tem_gb300 import _lib, imaging, synth
from tests.test_gpu_parity import FP32_TOL, FP64_TOL, setup_both

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = imaging.Context(0)
    yield c
    c.close()


def cell_of(n, voids=1):
    return synth.make_cell(*n, seed=11, n_voids=voids, void_radius=(3.0, 4.5))


def test_fp32_steps_about_the_renormalisation_rule(ctx):
    """Angles on both sides of 2 dz (b0 + bg + a) = 1: the image of six beside one of sixteen is the image alone."""
    t, _, x = setup_both(cell_of((6, 5, 6)), sg=0.0)
    G, _ = t.image_geometry(len(x))
    at = 1.0 / (2 * G.deltaz) - G.b0 - G.bg
    six, sixteen = np.linspace(0.9, 1.1, 6) * at, np.linspace(-1.2, 1.2, 16) * at
    assert (2 * G.deltaz * (G.b0 + G.bg + six[:2]) < 1).all() and (2 * G.deltaz * (G.b0 + G.bg + six[-2:]) > 1).all()
    want = ctx.image(G, x, six, flags=_lib.ST_FLAG_FP32)
    got = ctx.batch([(G, x, six), (G, x, sixteen)], _lib.ST_FLAG_FP32)
    assert np.array_equal(got[0], want)
    assert np.array_equal(got[1], ctx.image(G, x, sixteen, flags=_lib.ST_FLAG_FP32))
