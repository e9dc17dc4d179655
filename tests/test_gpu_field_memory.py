"""The field's sample workspace at its limits: an image or batch that runs in many ranges, down to one tile of
columns at a time, is the image of one range; without a workspace the general kernels compute it."""
import numpy as np
import pytest

from simulated_tem_gb300 import _lib, imaging, synth
from tests.test_gpu_parity import FP32_TOL, FP64_TOL

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def jobs_of(density):
    """Images of several depths and sizes, of four slices per step and (one voxel per a0 in depth) two."""
    out = []
    for n, M, n_prec in (((7, 6, 9), (4, 4), 1), ((5, 8, 4), (4, 4), 3), ((9, 6, 7), (4, 1), 1),
                          ((6, 6, 3), (3, 3), 1)):
        cell = synth.make_cell(*n, seed=5, n_voids=1, void_radius=(3.0, 4.0))
        t, x, _ = imaging.d2bi_condition(cell.a_super, synth.A0_FE, (0, 0, 1), (1, 1, 0), cell.pos, sg=0.01, M=M,
                                         density=density)
        G, aa = t.image_geometry(len(x), n_prec=n_prec)
        out.append((G, x, aa))
    return out


def batch(limit, jobs, flags):
    with pytest.MonkeyPatch.context() as m:
        if limit is not None:
            m.setenv("STEM_SAMPLE_BYTES", str(limit))
        c = imaging.Context(0)
    try:
        return c.batch(jobs, flags), c.stats().column_kernel, c.stats().n_launches
    finally:
        c.close()


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("density", [True, False])
def test_many_ranges_equal_one(fp32, density):
    jobs, flags = jobs_of(density), (_lib.ST_FLAG_FP32 if fp32 else 0) | _lib.ST_FLAG_AVERAGE
    want, kernel, launches = batch(None, jobs, flags)
    assert kernel == (2 if fp32 else 4)
    for limit in (1, 100_000, 1_000_000, "", "2G"):  # the last two are no numbers, and no bound
        got, k, n = batch(limit, jobs, flags)
        assert k == kernel and (n > launches or limit in (1_000_000, "", "2G"))
        for a, b in zip(got, want):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("fp32", [True, False])
def test_no_workspace_takes_the_general_kernels(fp32):
    jobs, flags = jobs_of(True), (_lib.ST_FLAG_FP32 if fp32 else 0) | _lib.ST_FLAG_AVERAGE
    want, _, _ = batch(None, jobs, flags)
    got, kernel, _ = batch(0, jobs, flags)
    assert kernel == (1 if fp32 else 3)
    for a, b in zip(got, want):
        assert np.abs(a - b).max() <= (FP32_TOL if fp32 else FP64_TOL)


def test_a_plan_keeps_its_contexts_bound():
    """The private contexts of a plan take the bound of the context that it is made from."""
    with pytest.MonkeyPatch.context() as m:
        m.setenv("STEM_SAMPLE_BYTES", "100000")
        c = imaging.Context(0)
    try:
        G, aa, x = jobs_of(False)[0]
        d_x = torch.from_numpy(x).cuda()
        img = torch.zeros((G.My, G.Mx), dtype=torch.float64, device="cuda")
        job = [(G, d_x.data_ptr(), len(x), aa, img.data_ptr())]
        stream = torch.cuda.current_stream().cuda_stream
        c.batch_device(job, _lib.ST_FLAG_FP32, stream)
        want, launches = img.clone(), c.stats().n_launches
        p = c.plan(job, _lib.ST_FLAG_FP32, stream)
        try:
            img.zero_()
            p.launch(stream)
            p.wait(stream)
            assert p.stats().n_launches == launches > 8
            assert torch.equal(img, want)
        finally:
            p.close()
    finally:
        c.close()
