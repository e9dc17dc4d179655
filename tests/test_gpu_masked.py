"""Tile-masked images: the wanted tiles are listed on the GPU, and the work and its split in depth follow their
number.  Whatever the mask, tile size, window, patch shape, slab capacity and workspace, the wanted tiles are the
plain image's to the last bit and the others zero."""
import numpy as np
import pytest

from simulated_tem_gb300 import _lib, imaging, synth

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def geometry(M=(4, 4), density=False, window=None):
    cell = synth.make_cell(9, 8, 7, seed=4, n_voids=1, void_radius=(3.0, 4.0))
    t, x, _ = imaging.d2bi_condition(cell.a_super, synth.A0_FE, (0, 0, 1), (1, 1, 0), cell.pos, sg=0.01, M=M,
                                     density=density)
    G, aa = t.image_geometry(len(x))
    if window:
        G.ix0, G.iy0, G.ix1, G.iy1 = window
    return G, aa, x


def check(c, G, aa, x, flags, mask, T):
    full = c.image(G, x, aa, flags=flags)
    kernel = c.stats().column_kernel
    img = torch.full((G.My, G.Mx), 3.0, dtype=torch.float64, device="cuda")
    d_x, d_mask = torch.from_numpy(x).cuda(), torch.from_numpy(mask).cuda()
    c.image_device_masked(G, d_x.data_ptr(), len(x), aa, flags, img.data_ptr(), d_mask.data_ptr(), T,
                          stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert c.stats().column_kernel == kernel == (2 if flags & _lib.ST_FLAG_FP32 else 4)
    sel = np.kron(mask, np.ones((T, T), dtype=np.uint8))[:G.My, :G.Mx].T.astype(bool)
    assert np.array_equal(img.cpu().numpy().T, np.where(sel, full, 0.0))


def mask_of(G, T, kind):
    shape = (-(-G.My // T), -(-G.Mx // T))
    m = np.zeros(shape, dtype=np.uint8)
    if kind == "one":
        m[-1, -1] = 1
    elif kind == "all":
        m[:] = 255
    elif kind != "none":
        m[:] = np.random.default_rng(int(100 * kind)).random(shape) < kind
    return m


@pytest.fixture(scope="module")
def ctx():
    c = imaging.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("kind", ["none", "one", "all", 0.1, 0.5])
@pytest.mark.parametrize("T", [8, 24])
def test_masks(ctx, fp32, kind, T):
    G, aa, x = geometry()
    check(ctx, G, aa, x, _lib.ST_FLAG_FP32 if fp32 else 0, mask_of(G, T, kind), T)


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("options", [dict(density=True), dict(M=(4, 1)), dict(window=(8, 4, 39, 47)),
                                     dict(window=(16, 20, 17, 30))])
def test_depths_windows_and_density(ctx, fp32, options):
    G, aa, x = geometry(**options)
    check(ctx, G, aa, x, (_lib.ST_FLAG_FP32 if fp32 else 0) | _lib.ST_FLAG_AVERAGE, mask_of(G, 8, 0.3), 8)


@pytest.mark.parametrize("variant", range(6))
def test_patch_shapes(variant):
    G, aa, x = geometry(window=(0, 4, 41, 48))
    c = imaging.Context(0)
    try:
        c.tune(variant)
        check(c, G, aa, x, _lib.ST_FLAG_FP32, mask_of(G, 8, 0.3), 8)
    finally:
        c.close()


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("env", [dict(STEM_RING_SLABS="192"), dict(STEM_RING_SLABS="256"),
                                 dict(STEM_SAMPLE_BYTES="40000")])
def test_slabs_and_ranges(fp32, env):
    G, aa, x = geometry()
    with pytest.MonkeyPatch.context() as m:
        for k, v in env.items():
            m.setenv(k, v)
        c = imaging.Context(0)
    try:
        for kind in ("none", "all", 0.3):
            check(c, G, aa, x, _lib.ST_FLAG_FP32 if fp32 else 0, mask_of(G, 8, kind), 8)
    finally:
        c.close()
