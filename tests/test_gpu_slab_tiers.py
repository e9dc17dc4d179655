"""Every tier of the slab ring's staging gives the same image, on both paths and with two or four slices per step, and
denser images than a tier holds move on to the next instead of the general kernel."""
import numpy as np
import pytest

from simulated_tem_gb300 import _lib, imaging, synth
from tests.test_gpu_parity import FP32_TOL, FP64_TOL

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

TIERS = ["128", "192", "256", "patch", "patch1024"]


def context(**env):
    with pytest.MonkeyPatch.context() as m:
        for k, v in env.items():
            m.setenv(k, v)
        return imaging.Context(0)


def condition(M, reps=1, n=(8, 7, 7), density=False):
    cell = synth.make_cell(*n, seed=4, n_voids=1, void_radius=(3.0, 4.0))
    pos = np.concatenate([cell.pos + 0.3 * k for k in range(reps)])
    t, x, _ = imaging.d2bi_condition(cell.a_super, synth.A0_FE, (0, 0, 1), (1, 1, 0), pos, sg=0.01, M=M, density=density)
    G, aa = t.image_geometry(len(x))
    return G, aa, x


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("M", [(4, 4), (4, 1)])
@pytest.mark.parametrize("density", [False, True])
def test_tiers_agree(fp32, M, density):
    G, aa, x = condition(M, density=density)
    flags = _lib.ST_FLAG_FP32 if fp32 else 0
    want = None
    for tier in TIERS:
        c = context(STEM_RING_SLABS=tier)
        try:
            got = c.image(G, x, aa, flags=flags)
            assert c.stats().column_kernel == (2 if fp32 else 4)
            stats = c.image(G, x, aa, flags=flags | _lib.ST_FLAG_STATS)
        finally:
            c.close()
        want = got if want is None else want
        assert np.array_equal(got, want) and np.array_equal(stats, want)


@pytest.mark.parametrize("M,reps", [((4, 4), 2), ((3, 3), 2), ((4, 4), 3), ((2, 2), 1), ((2, 2), 2), ((4, 1), 2),
                                    ((8, 1), 1), ((6, 6), 4)])
def test_dense_images_stay_on_the_ring(M, reps):
    """Up to 256 atoms per patch and slab, whatever the step's window holds."""
    G, aa, x = condition(M, reps, n=(14, 13, 9))
    c, general = context(), context(STEM_FP32_KERNEL="general", STEM_FP64_KERNEL="general")
    try:
        got = c.image(G, x, aa, flags=_lib.ST_FLAG_FP32)
        assert c.stats().column_kernel == 2
        assert np.abs(got - general.image(G, x, aa, flags=_lib.ST_FLAG_FP32)).max() <= FP32_TOL
        got = c.image(G, x, aa)
        assert c.stats().column_kernel == 4
        assert np.abs(got - general.image(G, x, aa)).max() <= FP64_TOL
    finally:
        c.close()
        general.close()


def test_two_slices_per_step_have_one_variant():
    """An image of deep voxels alone is not tuned, and reports variant 0 whatever was asked for."""
    cell = synth.make_cell(100, 100, 8, 13, n_voids=2, void_radius=(5.0, 8.0))
    t, x, _ = imaging.d2bi_condition(cell.a_super, synth.A0_FE, (0, 0, 1), (1, 1, 0), cell.pos, sg=0.01, M=(4, 1))
    G, aa = t.image_geometry(len(x))
    assert ((G.ix1 - G.ix0 + 7) // 8) * ((G.iy1 - G.iy0 + 3) // 4) >= 4096  # large enough to tune
    c = context()
    try:
        c.image(G, x, aa, flags=_lib.ST_FLAG_FP32)  # finds the slab tier
        launches = []
        for mode in (_lib.ST_TUNE_AUTO, _lib.ST_TUNE_OFF, 3):
            c.tune(mode)
            c.image(G, x, aa, flags=_lib.ST_FLAG_FP32)
            launches.append(c.stats().n_launches)
            assert c.stats().column_kernel == 2 and c.stats().ring_variant == 0
        assert len(set(launches)) == 1
    finally:
        c.close()
