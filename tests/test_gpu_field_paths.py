"""The field and integrator kernels where their paths change: pixel windows about the patches and tiles,
columns split in depth, equidistant atoms (exact nearest distances), angle counts about the integrators'
groups, and on both sides of the fixed-point integrator's rule; against the oracle."""
import numpy as np
import pytest

from simulated_tem_gb300 import _lib, imaging, synth
from tests.test_gpu_parity import FP32_TOL, FP64_TOL, oracle_patch, setup_both

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = imaging.Context(0)
    yield c
    c.close()


def cell_of(n, jitter=0.05, voids=1):
    return synth.make_cell(*n, seed=11, n_voids=voids, void_radius=(3.0, 4.5), jitter=jitter)


@pytest.mark.parametrize("n,jitter,n_prec,options", [
    ((8, 8, 6), 0.0, 1, dict(density=True, sg=0.01)),       # perfect lattice: ties everywhere
    ((8, 7, 6), 0.05, 1, dict(sg=0.5)),                     # steps too long for fixed point
    ((8, 7, 6), 0.05, 2, dict(sg=0.01, xig=1e6)),           # reflection too weak for fixed point
    ((8, 7, 6), 0.05, 1, dict(sg=0.01, xig=4e3)),           # on the rule's other side of that
    ((6, 9, 6), 0.05, 9, dict(sg=0.01, density=True)),      # two groups of eight angles
    ((5, 5, 40), 0.05, 1, dict(sg=0.005)),                  # few deep columns: split over warps
    ((6, 5, 3), 0.0, 1, dict(sg=0.0, density=True)),
])
def test_fp64_paths(ctx, n, jitter, n_prec, options):
    t, so, x = setup_both(cell_of(n, jitter), **options)
    G, aa = t.image_geometry(len(x), prec_angle=0.005, n_prec=n_prec)
    got = ctx.image(G, x, aa, flags=_lib.ST_FLAG_STATS | _lib.ST_FLAG_AVERAGE)
    st = ctx.stats()
    want, ost = oracle_patch(so, x, n_prec, 0.005)
    assert np.abs(got - want / n_prec).max() <= FP64_TOL
    assert st.n_kept == ost.n_kept and st.n_accepted == ost.n_accepted


@pytest.mark.parametrize("n,n_prec,options", [
    ((8, 7, 6), 1, dict(sg=0.01)),
    ((6, 9, 6), 2, dict(sg=0.01, density=True)),
    ((6, 9, 6), 9, dict(sg=0.0)),
    ((7, 5, 6), 33, dict(sg=0.01)),
    ((5, 5, 40), 1, dict(sg=0.005, density=True)),
    ((6, 5, 3), 1, dict(sg=0.0)),
])
def test_fp32_paths(ctx, n, n_prec, options):
    t, so, x = setup_both(cell_of(n), **options)
    G, aa = t.image_geometry(len(x), prec_angle=0.005, n_prec=n_prec)
    got = ctx.image(G, x, aa, flags=_lib.ST_FLAG_FP32 | _lib.ST_FLAG_AVERAGE)
    want, _ = oracle_patch(so, x, n_prec, 0.005)
    assert np.abs(got - want / n_prec).max() <= FP32_TOL


@pytest.fixture(scope="module")
def general():
    """A context that takes the general kernels (one column per thread, any cells)."""
    with pytest.MonkeyPatch.context() as m:
        m.setenv("STEM_FP64_KERNEL", "general")
        m.setenv("STEM_FP32_KERNEL", "general")
        c = imaging.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("density", [False, True])
def test_windows_equal_the_general_kernels(ctx, general, fp32, density):
    """Pixel windows (each with link cells of its own) about the patches of 8 x 4 and tiles of 16 x 8."""
    t, _, x = setup_both(cell_of((9, 10, 6)), sg=0.01, density=density)
    flags = _lib.ST_FLAG_FP32 if fp32 else 0
    for ix0, iy0, dx, dy in ((0, 0, 1, 1), (3, 2, 7, 3), (1, 5, 8, 4), (0, 1, 9, 5), (2, 0, 16, 8), (1, 1, 17, 9)):
        G, aa = t.window_geometry(len(x), ix0, iy0, dx, dy)
        got, want = ctx.image(G, x, aa, flags=flags), general.image(G, x, aa, flags=flags)
        assert np.abs(got - want).max() <= (FP32_TOL if fp32 else FP64_TOL)


@pytest.mark.parametrize("lattice,M", [("bcc", 2), ("bcc", 3), ("fcc", 2), ("fcc", 4), ("sc", 5)])
def test_coarse_voxels_and_dense_slabs(ctx, general, lattice, M):
    """Slices of up to a sigma (two per step in FP32) and every slab capacity, against the general kernels."""
    base = {"bcc": [[0, 0, 0], [0.5, 0.5, 0.5]], "sc": [[0, 0, 0]],
            "fcc": [[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]]}[lattice]
    n, a0 = np.array([10, 9, 8]), 3.6
    sites = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 1, 3)
    pos = (sites + np.array(base)).reshape(-1, 3) * a0
    pos = pos + np.random.default_rng(M).normal(0.0, 0.05, pos.shape)
    t, x, _ = imaging.d2bi_condition(np.diag(n * a0), a0, (0, 0, 1), (1, 1, 0) if lattice == "bcc" else (2, 0, 0), pos,
                                     sg=0.01, lattice=lattice, M=(M, M))
    G, aa = t.image_geometry(len(x))
    for flags, tol in ((_lib.ST_FLAG_FP32, FP32_TOL), (0, FP64_TOL)):
        assert np.abs(ctx.image(G, x, aa, flags=flags) - general.image(G, x, aa, flags=flags)).max() <= tol


@pytest.mark.parametrize("count", [1, 4, 24])
def test_batches_about_the_cell_scans_limit(ctx, count):
    """One block scans up to 16,384 cells; batches on both sides equal the single images."""
    torch = pytest.importorskip("torch")
    t, _, x = setup_both(cell_of((10, 10, 8)), sg=0.01)
    G, aa = t.image_geometry(len(x))
    want = ctx.image(G, x, aa, flags=_lib.ST_FLAG_FP32)
    xd = torch.from_numpy(x).to("cuda")
    out = torch.zeros((count, G.My, G.Mx), dtype=torch.float64, device="cuda")
    ctx.batch_device([(G, xd.data_ptr(), len(x), aa, out[i].data_ptr()) for i in range(count)], _lib.ST_FLAG_FP32,
                     torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for i in range(count):
        assert np.array_equal(out[i].cpu().numpy().T, want)
