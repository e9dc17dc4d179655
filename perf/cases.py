"""Performance cases of the imaging path: the calls a program that uses this package makes.

Each case names one kind of call and its sizes:

* image32 / image64: one condition on atoms resident on the GPU (``Context.image_device``),
  the FP32 path and the plain FP64 path;
* host64: one condition from host arrays (``Context.image``), the call the reference's
  Fortran host makes in place of its patch loop;
* sweep: a tomography series with beam precession, one ``batch_device`` call;
* cells: independent cells of uneven size, one ``batch_device`` call;
* blur: the PNG writer's Gaussian blur on a device image;
* lammps: the atom lines of a LAMMPS data file, parsed on the GPU;
* conv: one convolution layer of the corrector, forward (inference);
* conv_bwd: the gradients of such a layer (training).

Cells are bcc Fe as in the package's synthetic workloads (jitter, a screw dislocation along
z, spherical voids); the positions come from the seed.  The voxel grids, deviation
parameters and g-vectors are those of the tests and the benchmark.

The FP32 path computes single-precision intensities and stores them in the double image its
Fortran caller expects; the autotuner picks among tile shapes whose images agree to single
rounding.  ``run`` returns such images in the type they were computed in (float32), and the
FP64 path's in float64.
"""
import math
import random

import numpy as np
import torch

from simulated_tem_gb300 import _lib, imaging, synth
from simulated_tem_gb300 import nn as N

A0 = synth.A0_FE
SIGMA = A0 / 2
_shared = {}


def _context():
    """The program's one imaging context and the stream it works on."""
    if "ctx" not in _shared:
        _shared["ctx"] = imaging.Context(0)
        _shared["stream"] = torch.cuda.Stream()
    return _shared["ctx"], _shared["stream"]


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------

def listed():
    return [
        # the smallest cells people image (unit tests, quick looks): launches and latency
        dict(name="image32 1.6k atoms", kind="image32", nx=10, ny=10, nz=8, m=4, g="110", sg=0.01, n_prec=1,
             density=False),
        # the CPU-runnable configuration (40^3 cells, voids, density field)
        dict(name="image32 128k atoms density", kind="image32", nx=40, ny=40, nz=40, m=4, g="110", sg=0.01, n_prec=1,
             density=True),
        # the headline: a 1.2M-atom cell with a screw dislocation and voids, one dark field
        dict(name="image32 1.2M atoms", kind="image32", nx=100, ny=100, nz=60, m=4, g="110", sg=0.01, n_prec=1,
             density=False),
        # the reference-accurate path from host arrays, at the size of the reference's own test
        # (27,847 atoms, about 95^3 voxels), odd cell counts
        dict(name="host64 28k atoms", kind="host64", nx=23, ny=25, nz=24, m=4, g="200", sg=0.0074, n_prec=1,
             density=False),
        # the CPU-runnable configuration on the plain FP64 path
        dict(name="image64 128k atoms density", kind="image64", nx=40, ny=40, nz=40, m=4, g="110", sg=0.01, n_prec=1,
             density=True),
        # FP64 with beam precession (the path of -nPrec runs that are compared with the reference)
        dict(name="image64 16k atoms precession", kind="image64", nx=21, ny=20, nz=19, m=4, g="110", sg=0.01,
             n_prec=6, density=False),
        # tomography steps x two g-vectors with 16 precession angles each, one call
        dict(name="sweep 6 images x 16 angles", kind="sweep", nx=63, ny=60, nz=40, m=4, tilts=3, n_prec=16),
        # independent cells of 10k to 150k atoms, one call
        dict(name="cells 16 uneven", kind="cells", count=16, lo=10000, hi=150000, shapes=11),
        # the blur of a PNG of the headline cell at twice the pixel density
        dict(name="blur 1132x1131", kind="blur", nx=1132, ny=1131, t=6.97),
        # reading 300k atoms as LAMMPS' write_data prints them
        dict(name="lammps 300k atoms", kind="lammps", atoms=300000),
        # the decoder's first half-resolution layer on an 1132 x 1132 image
        dict(name="conv 568x568 192-64", kind="conv", b=1, h=568, w=568, cin=192, cout=64),
        # a half-resolution layer's gradients for a training batch of eight 512 x 512 crops
        dict(name="conv backward 8x256x256 64-64", kind="conv_bwd", b=8, h=256, w=256, cin=64, cout=64),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _voxels(c):
    """About the voxels of an image: the atoms' extents in the frame of (k, g) at m voxels per
    lattice constant."""
    m = c["m"]
    if c["g"] == "200":
        ex, ey = c["nx"], c["ny"]
    else:  # 110: the cell turned by 45 degrees
        ex = ey = (c["nx"] + c["ny"]) / math.sqrt(2)
    return ex * m * ey * m * c["nz"] * m


# layers of the corrector's network: (input channels, output channels, level)
LAYERS = [(16, 32, 0), (32, 32, 0), (32, 64, 1), (64, 64, 1), (64, 128, 2), (128, 128, 2), (128, 256, 3),
          (256, 256, 3), (384, 128, 2), (192, 64, 1), (96, 32, 0)]


def draw(rng):
    kind = rng.choice(["image32"] * 5 + ["image64"] * 2 + ["host64", "sweep", "cells", "blur", "lammps", "conv",
                                                              "conv_bwd"])
    if kind in ("image32", "image64", "host64"):
        most = 7.5e7 if kind == "image32" else 7.5e6
        while True:
            n = _log(rng, 8, 100)
            c = dict(kind=kind, nx=max(6, round(n * rng.uniform(0.7, 1.3))), ny=max(6, round(n * rng.uniform(0.7, 1.3))),
                     nz=max(6, round(_log(rng, 6, 70))), m=rng.choice([4, 4, 4, 4, 2, 3, 8]),
                     g=rng.choice(["110", "110", "200"]), sg=round(rng.uniform(-0.02, 0.02), 4),
                     n_prec=rng.choice([1, 1, 1, 1, 2, 5, 8, 16]) if kind == "image32" else rng.choice([1, 1, 1, 3]),
                     density=rng.random() < 0.35)
            if _voxels(c) * (1 + 0.05 * (c["n_prec"] - 1)) <= most and 2 * c["nx"] * c["ny"] * c["nz"] <= 1200000:
                return c
    if kind == "sweep":
        while True:
            n = _log(rng, 16, 63)
            c = dict(kind=kind, nx=max(10, round(n * rng.uniform(0.8, 1.2))), ny=max(10, round(n * rng.uniform(0.8, 1.2))),
                     nz=max(8, round(_log(rng, 8, 40))), m=4, tilts=rng.randint(2, 6),
                     n_prec=rng.choice([1, 4, 7, 16, 16]))
            if _voxels(dict(c, g="110")) * c["tilts"] <= 6e7:
                return c
    if kind == "cells":
        return dict(kind=kind, count=rng.randint(3, 16), lo=10000, hi=round(_log(rng, 20000, 150000)),
                    shapes=rng.randrange(1 << 20))
    if kind == "blur":
        return dict(kind=kind, nx=round(_log(rng, 60, 1130)), ny=round(_log(rng, 60, 1130)),
                    t=round(rng.uniform(1.0, 7.0), 2))
    if kind == "lammps":
        return dict(kind=kind, atoms=round(_log(rng, 2000, 300000)))
    cin, cout, level = rng.choice(LAYERS)
    if kind == "conv":
        side = 1100 if level == 0 else 560 >> (level - 1)
        return dict(kind=kind, b=1, h=round(_log(rng, 48, side)), w=round(_log(rng, 48, side)), cin=cin, cout=cout)
    side = 512 >> level
    if level == 0:
        return dict(kind=kind, b=rng.choice([1, 2]), h=side, w=side, cin=max(cin, 32), cout=cout)
    return dict(kind=kind, b=rng.choice([1, 2, 5, 8] if cin <= 128 else [1, 2, 3]), h=side, w=side, cin=cin, cout=cout)


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------

def _cell(nx, ny, nz, seed, voids, radius, screw):
    """A bcc cell (a_super, positions (N, 3) on the host): jitter of 0.05 A, a screw dislocation
    along z, spherical voids removed with the minimum-image distance.  Eight atoms sit at the
    cell's corners, so that the image box (the atoms' extents) does not depend on the jitter."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kw = dict(dtype=torch.float64, device="cuda")
    i, j, k = torch.meshgrid(torch.arange(nx, **kw), torch.arange(ny, **kw), torch.arange(nz, **kw), indexing="ij")
    corner = torch.stack([i, j, k], dim=-1).reshape(-1, 3)
    pos = torch.cat([corner, corner + 0.5]) * A0
    pos += 0.05 * torch.randn(pos.shape, generator=gen, **kw)
    box = torch.tensor([nx, ny, nz], **kw) * A0
    if screw:
        pos[:, 2] += A0 * torch.atan2(pos[:, 1] - box[1] / 2, pos[:, 0] - box[0] / 2) / (2 * math.pi)
    keep = torch.ones(len(pos), dtype=torch.bool, device="cuda")
    for _ in range(voids):
        c = torch.rand(3, generator=gen, **kw) * box
        r = radius[0] + (radius[1] - radius[0]) * torch.rand(1, generator=gen, **kw)
        d = pos - c
        d -= box * torch.round(d / box)
        keep &= (d * d).sum(dim=1) > r * r
    pos = pos[keep]
    pos[:8] = torch.cartesian_prod(*[torch.tensor([0.0, 1.0 - 1e-9], **kw)] * 3) * box
    return np.diag(box.cpu().numpy()), np.ascontiguousarray(pos.cpu().numpy())


def _g(name):
    return tuple(int(v) for v in name)


def _condition(c, seed):
    """The condition's geometry, wrapped atoms and precession parameters, as the package's
    set-up calls give them."""
    n = 2 * c["nx"] * c["ny"] * c["nz"]
    voids = 1 if n < 10000 else 8 if n < 500000 else 20
    small = min(c["nx"], c["ny"], c["nz"])
    radius = (4.0, 6.0) if small < 20 else (5.0, 12.0)
    a_super, pos = _cell(c["nx"], c["ny"], c["nz"], seed, voids, radius, not c["density"])
    t, x, _ = imaging.d2bi_condition(a_super, A0, (0, 0, 1), _g(c["g"]), pos, sg=c["sg"], M=(c["m"], c["m"]),
                                     density=c["density"])
    G, aa = t.image_geometry(len(x), prec_angle=0.005, n_prec=c["n_prec"])
    return G, x, aa


def _image_buffer(G):
    return torch.empty((G.My, G.Mx), dtype=torch.float64, device="cuda")


def _uneven_shapes(c):
    rng = random.Random(c["shapes"])
    out = []
    for _ in range(c["count"]):
        n = _log(rng, c["lo"], c["hi"])
        ax, ay = rng.uniform(0.5, 2.0), rng.uniform(0.5, 2.0)
        nz = max(6, round((n / 2 / (ax * ay)) ** (1 / 3)))
        nx = max(6, round(ax * nz))
        ny = max(6, round(n / 2 / (nx * nz)))
        out.append((nx, ny, nz, rng.randint(0, 10), rng.uniform(-0.02, 0.02)))
    return out


def _lammps_text(n, seed):
    """n atom lines as LAMMPS' write_data prints them, "id type x y z ix iy iz" with coordinates
    in %-1.16e, as a byte tensor on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    v = 280.0 * torch.rand((n, 3), generator=gen, dtype=torch.float64, device="cuda")
    neg = torch.rand((n, 3), generator=gen, device="cuda") < 0.002
    e = torch.floor(torch.log10(v)).clamp(-3, 2).to(torch.int64)
    mant = (v * torch.pow(torch.tensor(10.0, dtype=torch.float64, device="cuda"), (16 - e).double())).to(torch.int64)
    mant = mant.clamp(10 ** 16, 10 ** 17 - 1)
    mant = (mant // 64) * 64 + torch.randint(0, 64, (n, 3), generator=gen, device="cuda")
    mant = mant.clamp(10 ** 16, 10 ** 17 - 1)
    cols, masks = [], []

    def const(ch, mask=None):
        cols.append(torch.full((n,), ord(ch), dtype=torch.uint8, device="cuda"))
        masks.append(torch.ones(n, dtype=torch.bool, device="cuda") if mask is None else mask)

    ident = torch.arange(1, n + 1, device="cuda")
    width = len(str(n))
    for p in range(width - 1, -1, -1):
        cols.append((ident // 10 ** p % 10 + 48).to(torch.uint8))
        masks.append(ident >= 10 ** p)
    const(" ")
    const("1")
    for a in range(3):
        const(" ")
        const("-", neg[:, a])
        for p in range(16, -1, -1):
            cols.append((mant[:, a] // 10 ** p % 10 + 48).to(torch.uint8))
            masks.append(torch.ones(n, dtype=torch.bool, device="cuda"))
            if p == 16:
                const(".")
        const("e")
        cols.append(torch.where(e[:, a] < 0, ord("-"), ord("+")).to(torch.uint8))
        masks.append(torch.ones(n, dtype=torch.bool, device="cuda"))
        const("0")
        cols.append((e[:, a].abs() + 48).to(torch.uint8))
        masks.append(torch.ones(n, dtype=torch.bool, device="cuda"))
    for ch in " 0 0 0\n":
        const(ch)
    return torch.stack(cols, dim=1)[torch.stack(masks, dim=1)].contiguous()


def _bf16(shape, gen, std=1.0, relu=False):
    t = torch.randn(shape, generator=gen, dtype=torch.float32, device="cuda") * std
    return (t.clamp_(min=0) if relu else t).to(torch.bfloat16)


def prepare(case, seed):
    kind = case["kind"]
    ctx, stream = _context()
    if kind in ("image32", "image64"):
        G, x, aa = _condition(case, seed)
        flags = _lib.ST_FLAG_AVERAGE | (_lib.ST_FLAG_FP32 if kind == "image32" else 0)
        s = dict(case=case, G=G, aa=aa, n=len(x), x=torch.from_numpy(x).cuda(), img=_image_buffer(G), flags=flags)
    elif kind == "host64":
        G, x, aa = _condition(case, seed)
        s = dict(case=case, G=G, aa=aa, x=x, flags=_lib.ST_FLAG_AVERAGE)
    elif kind == "sweep":
        a_super, pos = _cell(case["nx"], case["ny"], case["nz"], seed, 8, (5.0, 12.0), True)
        d_x, specs, conds = imaging.d2bi_sweep(ctx, a_super, A0, (0, 0, 1), [(1, 1, 0), (2, 0, 0)], pos,
                                               n_tomo=case["tilts"], tomo_angle=20.0, prec_angle=0.005,
                                               n_prec=case["n_prec"], sg=0.01)
        specs = specs[:2 * case["tilts"]]
        imgs = [_image_buffer(G) for G, _ in specs]
        jobs = [(G, d_x.data_ptr(), len(pos), aa, im.data_ptr()) for (G, aa), im in zip(specs, imgs)]
        s = dict(case=case, jobs=jobs, imgs=imgs, xs=[d_x], conds=conds)
    elif kind == "cells":
        jobs, imgs, xs, conds = [], [], [], []
        for i, (nx, ny, nz, voids, sg) in enumerate(_uneven_shapes(case)):
            a_super, pos = _cell(nx, ny, nz, seed * 64 + i, voids, (4.0, 12.0), False)
            t, x, _ = imaging.d2bi_condition(a_super, A0, (0, 0, 1), (1, 1, 0), pos, sg=sg)
            G, aa = t.image_geometry(len(x))
            xs.append(torch.from_numpy(x).cuda())
            imgs.append(_image_buffer(G))
            jobs.append((G, xs[-1].data_ptr(), len(x), aa, imgs[-1].data_ptr()))
            conds.append(t)
        s = dict(case=case, jobs=jobs, imgs=imgs, xs=xs, conds=conds)
    elif kind == "blur":
        # an image's values: a mean level, a few per cent of pixel noise and a smooth variation
        gen = torch.Generator(device="cuda").manual_seed(seed)
        nx, ny = case["nx"], case["ny"]
        img = 0.3 + 0.02 * torch.randn((ny, nx), generator=gen, dtype=torch.float64, device="cuda")
        p = torch.rand(4, generator=gen, dtype=torch.float64, device="cuda")
        yy = torch.arange(ny, dtype=torch.float64, device="cuda")[:, None]
        xx = torch.arange(nx, dtype=torch.float64, device="cuda")[None, :]
        img += 0.2 * torch.sin(0.02 * xx + 6.28 * p[0]) * torch.cos(0.03 * p[1] * yy + 6.28 * p[2])
        s = dict(case=case, img=img, out=torch.empty_like(img))
    elif kind == "lammps":
        text = _lammps_text(case["atoms"], seed)
        s = dict(case=case, text=text, x=torch.zeros((case["atoms"], 3), dtype=torch.float64, device="cuda"),
                 types=torch.zeros(case["atoms"], dtype=torch.int32, device="cuda"))
    else:
        gen = torch.Generator(device="cuda").manual_seed(seed)
        b, h, w, cin, cout = (case[k] for k in ("b", "h", "w", "cin", "cout"))
        x = _bf16((b, h, w, cin), gen, relu=True)
        wt = _bf16((cout, 9, cin), gen, std=math.sqrt(2.0 / (9 * cin)))
        s = dict(case=case, x=x, w=wt)
        if kind == "conv":
            s["bias"] = 0.1 * torch.randn(cout, generator=gen, dtype=torch.float32, device="cuda")
        else:
            s["g"] = _bf16((b, h, w, cout), gen, std=1e-3)
            s["flipped"] = N.weight_flip(wt)
            s["gw"] = torch.zeros((cout, 9, cin), dtype=torch.float32, device="cuda")
            s["gb"] = torch.zeros(cout, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------

def run(s):
    kind = s["case"]["kind"]
    ctx, stream = _context()
    if kind == "host64":
        return ctx.image(s["G"], s["x"], s["aa"], flags=s["flags"])
    if kind in ("conv", "conv_bwd"):  # torch's current stream
        if kind == "conv":
            return N.conv2d(s["x"], s["w"], s["bias"], relu=True)
        N.zero_(s["gw"])
        N.zero_(s["gb"])
        N.conv2d_wgrad(s["x"], s["g"], 9, s["gw"])
        N.bias_grad(s["g"], s["gb"])
        return {"gx": N.conv2d(s["g"], s["flipped"], mask=s["x"]), "gw": s["gw"], "gb": s["gb"]}
    with torch.cuda.stream(stream):
        st = stream.cuda_stream
        if kind in ("image32", "image64"):
            ctx.image_device(s["G"], s["x"].data_ptr(), s["n"], s["aa"], s["flags"], s["img"].data_ptr(), stream=st)
            return s["img"].float() if kind == "image32" else s["img"]
        if kind in ("sweep", "cells"):
            ctx.batch_device(s["jobs"], _lib.ST_FLAG_FP32 | _lib.ST_FLAG_AVERAGE, stream=st)
            return [im.float() for im in s["imgs"]]
        if kind == "blur":
            ny, nx = s["img"].shape
            ctx.blur_device(s["img"].data_ptr(), nx, ny, s["case"]["t"], s["out"].data_ptr(), stream=st)
            return s["out"]
        bad = ctx.parse_atoms_device(s["text"].data_ptr(), s["text"].numel(), s["case"]["atoms"], s["x"].data_ptr(),
                                     s["types"].data_ptr(), stream=st)
        return {"x": s["x"], "types": s["types"], "bad": bad}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------

def _image_work(atoms, voxels, pixels, n_prec, density):
    """Bytes: positions in, image out.  Operations: per neighbour within 3 sigma a weight
    times a phasor (12), per voxel the normalisation (6) and the density (10), per voxel and
    angle half an RK4 double step (90)."""
    pairs = 28.2 * voxels
    return {"bytes": 24.0 * atoms + 8.0 * pixels,
            "flops": 12.0 * pairs + voxels * (6.0 + (10.0 if density else 0.0) + 90.0 * n_prec)}


def work(case):
    kind = case["kind"]
    if kind in ("image32", "image64", "host64"):
        v = _voxels(case)
        return _image_work(2 * case["nx"] * case["ny"] * case["nz"], v, v / (case["nz"] * case["m"]), case["n_prec"],
                           case["density"])
    if kind == "sweep":
        v = sum(_voxels(dict(case, g=g)) for g in ("110", "200")) * case["tilts"]
        return _image_work(2 * case["nx"] * case["ny"] * case["nz"], v, v / (4 * case["nz"]), case["n_prec"], False)
    if kind == "cells":
        total = {"bytes": 0.0, "flops": 0.0}
        for nx, ny, nz, _, _ in _uneven_shapes(case):
            v = _voxels(dict(nx=nx, ny=ny, nz=nz, m=4, g="110"))
            w = _image_work(2 * nx * ny * nz, v, v / (4 * nz), 1, False)
            total = {k: total[k] + w[k] for k in total}
        return total
    if kind == "blur":
        n = case["nx"] * case["ny"]
        return {"bytes": 16.0 * n, "flops": 4.0 * n * (2 * max(5, math.ceil(5 * case["t"])) + 1)}
    if kind == "lammps":
        return {"bytes": case["atoms"] * (84.0 + 28.0), "flops": 0.0}
    b, h, w, cin, cout = (case[k] for k in ("b", "h", "w", "cin", "cout"))
    fma = 2.0 * b * h * w * 9 * cin * cout
    if kind == "conv":
        return {"bytes": 2.0 * (b * h * w * (cin + cout) + 9 * cin * cout) + 4 * cout, "flops": fma}
    return {"bytes": 2.0 * (b * h * w * (2 * cin + cout) + 9 * cin * cout) + 4.0 * (9 * cin * cout + cout),
            "flops": 2 * fma}


# ------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------

def _field(G, x):
    """The voxel sums of a condition in FP64, (Mz, My, Mx): real and imaginary part of
    sum exp(-r^2 / 2 sigma^2) exp(i g.y) over the atoms within 3 sigma, and the smallest r^2.
    The atoms' copies that lie in the link-cell box count, the box is periodic, and an atom
    counts for the voxels whose link cell is its own or one of the 26 around it (z cells can be
    a little shorter than 3 sigma).  Every atom adds itself to the voxels around it."""
    kw = dict(dtype=torch.float64, device="cuda")
    Mx, My, Mz = G.Mx, G.My, G.Mz
    RU = torch.tensor(list(G.RU), **kw).view(3, 3).T
    delta, lcd, g = (torch.tensor(list(v), **kw) for v in (G.delta, G.lc_delta, G.g))
    cell = torch.tensor([G.a_col[0], G.a_col[4], G.a_col[8]], **kw)
    icell = torch.tensor([G.ia_col[0], G.ia_col[4], G.ia_col[8]], **kw)
    vox = [G.a_vox[0], G.a_vox[4], G.a_vox[8]]
    box = cell * torch.tensor([G.Ex, G.Ey, G.Ez], **kw)
    cut = 3 * G.sigma
    parts = []
    for n in range(G.nuvw):
        u = x + torch.tensor([G.Ruvw[3 * n + k] for k in range(3)], **kw)
        y = (u[:, None, :] * RU).sum(dim=2) + delta
        z = y - lcd
        inside = ((z >= 0) & (z < box)).all(dim=1)
        parts.append(torch.cat([z[inside], (y[inside] * g).sum(dim=1, keepdim=True), torch.floor(z[inside] * icell)], dim=1))
    p = torch.cat(parts)
    count = (G.Ex, G.Ey, G.Ez)
    home = []  # a voxel's link cell along each axis
    for a in range(3):
        i = torch.arange((Mx, My, Mz)[a], **kw)
        home.append(torch.floor(icell[a] * (vox[a] * i - lcd[a])))
    for a in range(3):  # periodic copies within the cutoff of the voxels
        lo, hi = -lcd[a] - cut, -lcd[a] + vox[a] * ((Mx, My, Mz)[a] - 1) + cut
        out = [p]
        for sgn in (-1, 1):
            q = p.clone()
            q[:, a] += sgn * box[a]
            q[:, 4 + a] += sgn * count[a]
            out.append(q)
        p = torch.cat(out)
        p = p[(p[:, a] >= lo) & (p[:, a] <= hi)]
    y = p[:, :3] + lcd  # relative to voxel (0, 0, 0)
    cosp, sinp = torch.cos(p[:, 3]), torch.sin(p[:, 3])
    base, d2, ew = [], [], []
    reach = []
    for a in range(3):
        r = int(math.ceil(cut / vox[a])) + 1
        b = torch.floor(y[:, a] / vox[a]).to(torch.int64)
        off = torch.arange(-r, r + 1, device="cuda")
        d = y[:, a, None] - (b[:, None] + off).double() * vox[a]
        base.append(b)
        reach.append(r)
        d2.append((d * d).T.contiguous())
        ew.append(torch.exp(-(d * d) / (2 * G.sigma * G.sigma)).T.contiguous())
    n = Mx * My * Mz
    sr, si = torch.zeros(n + 1, **kw), torch.zeros(n + 1, **kw)
    rm = torch.full((n + 1,), 3.0e38, **kw) if G.useDensity else None
    for i in range(2 * reach[0] + 1):
        ix = base[0] + (i - reach[0])
        ax = d2[0][i] <= cut * cut
        ax &= (ix >= 0) & (ix < Mx)
        ax &= (home[0][ix.clamp(0, Mx - 1)] - p[:, 4]).abs() <= 1
        for j in range(2 * reach[1] + 1):
            iy = base[1] + (j - reach[1])
            h = d2[0][i] + d2[1][j]
            ay = (h <= cut * cut) & (iy >= 0) & (iy < My)
            ay &= (home[1][iy.clamp(0, My - 1)] - p[:, 5]).abs() <= 1
            sel = torch.nonzero(ax & ay)[:, 0]
            if not len(sel):
                continue
            h = h[sel]
            col = ix[sel] + Mx * iy[sel]
            w = ew[0][i][sel] * ew[1][j][sel]
            wc, ws, bz, cz = w * cosp[sel], w * sinp[sel], base[2][sel], p[sel, 6]
            for k in range(2 * reach[2] + 1):
                iz = bz + (k - reach[2])
                r2 = h + d2[2][k][sel]
                ok = (r2 <= cut * cut) & (iz >= 0) & (iz < Mz)
                ok &= (home[2][iz.clamp(0, Mz - 1)] - cz).abs() <= 1
                at = torch.where(ok, col + (Mx * My) * iz, n)
                e = torch.where(ok, ew[2][k][sel], 0.0)
                sr.index_add_(0, at, wc * e)
                si.index_add_(0, at, ws * e)
                if rm is not None:
                    rm.scatter_reduce_(0, at, r2, "amin")
    shape = (Mz, My, Mx)
    return sr[:n].view(shape), si[:n].view(shape), None if rm is None else rm[:n].view(shape)


def _image_exact(G, x, aa):
    """The image of a condition in FP64: the two-beam equations integrated down every column
    with the reference's RK4 double steps, averaged over the precession angles."""
    sr, si, rm = _field(G, x)
    mag = torch.sqrt(sr * sr + si * si).clamp(min=1e-16)
    xr, xi = sr / mag, si / mag
    del sr, si, mag
    if rm is not None:
        s = torch.sqrt(rm) / G.sigma - 1.0
        rho = 1.0 - s * s * s * (10.0 - 15.0 * s + 6.0 * s * s)
        rho = torch.where(rm < G.sigma ** 2, 1.0, torch.where(rm > 4 * G.sigma ** 2, 0.0, rho))
    else:
        rho = torch.ones((G.Mz, 1, 1), dtype=torch.float64, device="cuda")
    dz = G.deltaz
    img = torch.zeros(xr.shape[1:], dtype=torch.float64, device="cuda")
    for a in [float(v) for v in aa]:
        p = torch.zeros((2,) + xr.shape[1:], dtype=torch.complex128, device="cuda")
        p[0] = 1.0

        def deriv(k, q):
            k = k % G.Mz  # the column closes on its first sample
            c0 = G.b0 * rho[k]
            cg = G.bg * rho[k] * torch.complex(xr[k], xi[k])
            return torch.stack([1j * (c0 * q[0] + cg * q[1]), 1j * (torch.conj(cg) * q[0] + (c0 + a) * q[1])])

        for k in range(0, G.Mz - 1, 2):
            k1 = deriv(k, p)
            k2 = deriv(k + 1, p + dz * k1)
            k3 = deriv(k + 1, p + dz * k2)
            k4 = deriv(k + 2, p + 2 * dz * k3)
            p = p + (dz / 3) * (k1 + 2 * k2 + 2 * k3 + k4)
            p = p / torch.sqrt((p.real ** 2 + p.imag ** 2).sum(dim=0))
        img += p[1].real ** 2 + p[1].imag ** 2
    return img / len(aa)


def _conv_exact(x, w, pad=1):
    """A 3 x 3 convolution in FP64: x (B, H, W, C), w (Cout, 9, C); (B, H, W, Cout)."""
    b, h, wd, c = x.shape
    xp = torch.zeros((b, h + 2, wd + 2, c), dtype=torch.float64, device="cuda")
    xp[:, 1:-1, 1:-1] = x.double()
    out = torch.zeros((b, h, wd, w.shape[0]), dtype=torch.float64, device="cuda")
    for t in range(9):
        out += xp[:, t // 3:t // 3 + h, t % 3:t % 3 + wd] @ w[:, t].double().T
    return out


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind in ("image32", "image64"):
        return _image_exact(s["G"], s["x"], s["aa"])
    if kind == "host64":
        return _image_exact(s["G"], torch.from_numpy(s["x"]).cuda(), s["aa"]).T.cpu().numpy()
    if kind in ("sweep", "cells"):
        xs = s["xs"] if kind == "cells" else s["xs"] * len(s["jobs"])
        return [_image_exact(job[0], x, job[3]) for job, x in zip(s["jobs"], xs)]
    if kind == "blur":
        t = case["t"]
        nk = max(5, math.ceil(5 * t))
        k = torch.arange(-nk, nk + 1, dtype=torch.float64, device="cuda")
        k = torch.exp(-k * k / (2 * t * t))
        v = s["img"]
        for axis in (1, 0):
            n = v.shape[axis]
            i = torch.arange(n, device="cuda")
            num, den = torch.zeros_like(v), torch.zeros(n, dtype=torch.float64, device="cuda")
            for j in range(-nk, nk + 1):
                ok = (i + j >= 0) & (i + j < n)
                w = torch.where(ok, k[j + nk], 0.0)
                u = v.index_select(axis, (i + j).clamp(0, n - 1))
                num += u * (w[None, :] if axis == 1 else w[:, None])
                den += w
            v = num / (den[None, :] if axis == 1 else den[:, None])
        return v
    if kind == "lammps":
        vals = bytes(s["text"].cpu().numpy()).split()
        x = np.array([float(v) for i, v in enumerate(vals) if 2 <= i % 8 <= 4]).reshape(-1, 3)
        return {"x": torch.from_numpy(x), "types": None, "bad": None}
    if kind == "conv":
        return (_conv_exact(s["x"], s["w"]) + s["bias"].double()).clamp(min=0)
    b, h, w, cin, cout = (case[k] for k in ("b", "h", "w", "cin", "cout"))
    g = s["g"].double()
    gx = _conv_exact(s["g"], torch.flip(s["w"], dims=[1]).permute(2, 1, 0)) * (s["x"] > 0)
    xp = torch.zeros((b, h + 2, w + 2, cin), dtype=torch.float64, device="cuda")
    xp[:, 1:-1, 1:-1] = s["x"].double()
    gw = torch.stack([g.reshape(-1, cout).T @ xp[:, t // 3:t // 3 + h, t % 3:t % 3 + w].reshape(-1, cin)
                      for t in range(9)], dim=1)
    return {"gx": gx, "gw": gw, "gb": g.sum(dim=(0, 1, 2))}
