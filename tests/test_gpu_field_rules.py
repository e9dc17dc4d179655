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


@pytest.fixture(scope="module")
def general():
    """A context that takes the general kernels (one column per thread, any cells)."""
    with pytest.MonkeyPatch.context() as m:
        m.setenv("STEM_FP64_KERNEL", "general")
        m.setenv("STEM_FP32_KERNEL", "general")
        c = imaging.Context(0)
    yield c
    c.close()


def dilute(density, n_prec=1, **options):
    """A dilute gas in a deep box."""
    a0 = synth.A0_FE
    box = np.array([9, 8, 14]) * a0
    pos = np.random.default_rng(3).uniform(0.0, 1.0, (70, 3)) * box
    pos[:8] = np.array([[i, j, k] for i in (0, 1 - 1e-9) for j in (0, 1 - 1e-9) for k in (0, 1 - 1e-9)]) * box
    t, x, _ = imaging.d2bi_condition(np.diag(box), a0, (0, 0, 1), (1, 1, 0), pos, density=density,
                                     **{"sg": 0.01, **options})
    G, aa = t.image_geometry(len(x), prec_angle=0.005, n_prec=n_prec)
    return G, aa, x


@pytest.mark.parametrize("density", [False, True])
@pytest.mark.parametrize("n_prec", [1, 5])
def test_fp64_sparse_columns(ctx, general, density, n_prec):
    """A dilute gas in a deep box: most columns hold a weak field or none, down to the rim of one atom's density.
    Each intensity is as accurate, relative to itself, as the general kernel's in FP64."""
    G, aa, x = dilute(density, n_prec)
    got, want = ctx.image(G, x, aa), general.image(G, x, aa)
    assert ctx.stats().column_kernel == 4 and general.stats().column_kernel == 3
    assert (want < 1e-12).any() or not density
    assert (want > 1e-3).any()
    # 40 double steps and sums of a few terms: some tens of units of 2^-53
    assert (np.abs(got - want) <= 1e-12 * want + 1e-36).all()


@pytest.mark.parametrize("fp32", [False, True])
def test_sparse_image_beside_one_with_density(ctx, fp32):
    """An image without the density field in a batch with one that has it is the image alone, weak columns included
    (a reflection that lets one atom's edge reach a few thousandths)."""
    flags = _lib.ST_FLAG_FP32 if fp32 else 0
    plain, dens = (dilute(d, sg=0.002, xig=1900.0) for d in (False, True))
    G, aa, _ = plain
    assert 32 * G.bg >= abs(aa[0]) and G.Mz * G.deltaz * G.bg >= 1 / 16
    got = ctx.batch([(g[0], g[2], g[1]) for g in (plain, dens)], flags)
    assert ((got[0] > 0) & (got[0] < 2.0 ** -13)).any()
    for image, (G, aa, x) in zip(got, (plain, dens)):
        assert np.array_equal(image, ctx.image(G, x, aa, flags=flags))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_fp64_reflections_that_are_not_finite(ctx, general, axis, bad):
    """A g-vector that is not finite gives an image that is not, as the general kernel says."""
    t, _, x = setup_both(cell_of((6, 5, 5)), sg=0.01)
    G, aa = t.image_geometry(len(x))
    G.g[axis] = bad
    got, want = ctx.image(G, x, aa), general.image(G, x, aa)
    assert np.isnan(want).any()
    assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.parametrize("side,kernel", [(20.0, 4), (35.0, 4), (40.0, 3), (110.0, 3)])
def test_fp64_coarse_voxels_of_a_dilute_gas(ctx, general, side, kernel):
    """Voxels far beyond a lattice constant, a few atoms about each: the distances to a patch's reference cell grow
    until FP32 no longer decides (and the cells until their numbers leave a byte)."""
    t, _, x = setup_both(cell_of((6, 5, 5)), sg=0.01)
    G, aa = t.image_geometry(len(x))
    vox, n, cell = (side, 1.0, 1.0), (8, 4, 8), 3.2
    count = [int(np.ceil(vox[i] * (n[i] - 1) / cell)) + 3 for i in range(3)]
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(-1.5, 1.5, (12, 3)) + [side * i, 1.5, 3.5] for i in range(n[0])])
    x[:, 2] += rng.uniform(-3.0, 3.0, len(x))
    G.sigma, G.nuvw, G.useDensity, G.nMax0 = 1.0, 1, 0, 0
    G.Mx, G.My, G.Mz = n
    G.ix0, G.ix1, G.iy0, G.iy1 = 0, n[0], 0, n[1]
    G.Ex, G.Ey, G.Ez = count
    for k in range(9):
        i, diag = k // 3, k % 4 == 0
        G.RU[k] = 1.0 if diag else 0.0
        G.a_col[k] = cell if diag else 0.0
        G.ia_col[k] = 1.0 / cell if diag else 0.0
        G.a_vox[k] = vox[i] if diag else 0.0
    for k in range(3):
        G.delta[k] = G.Ruvw[k] = 0.0
        G.lc_delta[k] = -cell
        G.g[k] = 0.7 * k
    G.deltaz = 1.0
    got, want = ctx.image(G, x, aa), general.image(G, x, aa)
    assert ctx.stats().column_kernel == kernel and ctx.stats().n_kept == len(x)
    assert (want > 1e-4).sum() >= 20
    assert np.abs(got - want).max() <= FP64_TOL


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("density", [False, True])
def test_small_windows_on_the_field_kernels(ctx, general, fp32, density):
    """Pixel windows smaller than a patch, of a patch, of a tile and one more, in the whole image's link cells (a
    geometry made for a small window has cells too narrow for the field kernels)."""
    t, _, x = setup_both(cell_of((9, 10, 6)), sg=0.01, density=density)
    G, aa = t.image_geometry(len(x))
    flags = _lib.ST_FLAG_FP32 if fp32 else 0
    for ix0, iy0, dx, dy in ((0, 0, 1, 1), (3, 2, 7, 3), (1, 5, 8, 4), (0, 1, 9, 5), (2, 0, 16, 8), (1, 1, 17, 9),
                             (G.Mx - 1, G.My - 1, 1, 1), (G.Mx - 9, 0, 9, G.My)):
        G.ix0, G.ix1, G.iy0, G.iy1 = ix0, ix0 + dx, iy0, iy0 + dy
        got, want = ctx.image(G, x, aa, flags=flags), general.image(G, x, aa, flags=flags)
        assert ctx.stats().column_kernel == (2 if fp32 else 4) and general.stats().column_kernel == (1 if fp32 else 3)
        assert np.abs(got - want).max() <= (FP32_TOL if fp32 else FP64_TOL)
        inside = np.zeros(got.shape, dtype=bool)
        inside[ix0:ix0 + dx, iy0:iy0 + dy] = True
        assert (got[inside] != 0).any() and not got[~inside].any()


@pytest.mark.parametrize("n_prec", [1, 3])
def test_steps_long_enough_to_renormalise_each(ctx, general, n_prec):
    """2 dz (b0 + bg + |a|) of 1 and more: both integrators renormalise after every double step."""
    t, _, x = setup_both(cell_of((6, 5, 6)), sg=0.0)
    G, _ = t.image_geometry(len(x))
    aa = (np.array([1.05, -1.2, 1.4])[:n_prec]) / (2 * G.deltaz)
    assert (2 * G.deltaz * (G.b0 + G.bg + np.abs(aa)) >= 1).all()
    for flags, tol in ((_lib.ST_FLAG_FP32, FP32_TOL), (0, FP64_TOL)):
        got, want = ctx.image(G, x, aa, flags=flags), general.image(G, x, aa, flags=flags)
        assert ctx.stats().column_kernel == (2 if flags else 4)
        assert np.abs(got - want).max() <= tol * n_prec
