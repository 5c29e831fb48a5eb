"""Workloads of the projector, as a program that uses the framework runs them.

Every case is a geometry (a cube of voxels spanning 3 solar radii per axis and
a trajectory of conic views around it) plus the entry point that is called on
it.  The sizes are the framework's own workloads: the plain reconstruction
(64^3, 60 views of 128^2), the large one (256^3, 360 views of 512^2), the
time-dependent one (128^3 x 28 frames, 784 views of 256^2), packs of uneven
jobs, and the small / non-square / inclined geometries of the test-suite.

Operations (``op``):

* ``dropin_pj``  -- ``tomograpy_gb300.projector`` on CUDA tensors with headers;
* ``pj``, ``bpj`` -- ``lo_wrapper.siddon_lo(...).project`` / ``.backproject``;
* ``bpj_det``    -- the bitwise reproducible backprojection;
* ``pj4``, ``bpj4`` -- the 4-D operator (views mapped to cube frames);
* ``grad``       -- the differentiable projector: y = P x and the gradient of
  1/2 |P x - y0|^2;
* ``normal64``   -- P then P^T in float64 (the reference's default type);
* ``packed``     -- one packed launch per direction over several uneven jobs;
* ``cg``         -- conjugate gradients on P^T P + lam I (a whole solve).
"""
import math

import numpy as np
import torch

import tomograpy_gb300 as tg
from tomograpy_gb300 import autograd, batch, cg, lo_wrapper

EDGES = (32, 48, 64, 96, 128, 160, 192)     # cube edges of the uneven jobs
SIDES = (64, 128, 256)                      # their image sides
CG_ITERS = 4
CG_LAM = 1e-2


def _case(name, op, n, T, N, **kw):
    n = (n,) * 3 if isinstance(n, int) else tuple(n)
    N = (N,) * 2 if isinstance(N, int) else tuple(N)
    c = dict(op=op, n0=n[0], n1=n[1], n2=n[2], T=T, N1=N[0], N2=N[1], d=215.0, lon0=0.0, lon1=math.pi,
             lat=0.0, rol=0.0, sun=True, mask=False, frames=1)
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    two_pi = 2.0 * math.pi
    return [
        # the smallest call: the drop-in function on an integration-test size,
        # where the host path and the launches are what a user waits for
        _case("dropin24_pj", "dropin_pj", 24, 8, 32, lon0=0.1, lon1=3.0),
        # the plain reconstruction's projector and its adjoint
        _case("plain64_pj", "pj", 64, 60, 128),
        _case("plain64_bpj", "bpj", 64, 60, 128),
        # a whole small solve on the plain geometry
        _case("plain64_cg", "cg", 64, 60, 128),
        # the largest workload: one pass over a full orbit
        _case("recon256_pj", "pj", 256, 360, 512, lon1=two_pi),
        _case("recon256_bpj", "bpj", 256, 360, 512, lon1=two_pi),
        # the time-dependent workload, both directions
        _case("frames128_pj4", "pj4", 128, 784, 256, lon1=two_pi, frames=28),
        _case("frames128_bpj4", "bpj4", 128, 784, 256, lon1=two_pi, frames=28),
        # views from off the equator and rolled, odd non-square images, an
        # anisotropic cube and a pixel mask: what real ephemerides give
        _case("inclined_grad", "grad", (100, 84, 61), 45, (121, 90), d=190.0, lon0=0.2, lon1=4.4, lat=0.12,
              rol=0.3, mask=True),
        # bitwise reproducible backprojection
        _case("det96_bpj", "bpj_det", 96, 90, 192, lon0=0.3, lon1=5.0),
        # uneven jobs in one launch per direction
        _case("uneven6_packed", "packed", 64, 24, 128, jobs=6, jseed=3),
        # double precision
        _case("plain48_normal64", "normal64", 48, 12, 64, lon0=0.1, lon1=3.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["dropin_pj", "pj", "bpj", "pj", "bpj", "bpj_det", "pj4", "bpj4", "grad", "normal64", "packed",
                     "cg"])
    d = rng.uniform(150.0, 230.0)
    lon0 = rng.uniform(0.01, 1.0)
    kw = dict(d=d, lon0=lon0, lon1=lon0 + rng.uniform(1.5, 5.5), sun=rng.random() < 0.75)
    if rng.random() < 0.3 and op != "packed":      # off the equator
        kw.update(lat=rng.uniform(-0.13, 0.13), rol=rng.uniform(-0.4, 0.4))
    if op == "packed":
        return _case(None, op, 64, rng.randint(8, 48), 128, jobs=rng.randint(3, 10), jseed=rng.randint(10, 9999),
                     d=d, lon0=lon0, lon1=lon0 + 3.0)
    top_n, top_rays = {"dropin_pj": (64, 1e6), "normal64": (64, 2e5), "cg": (96, 2e6), "bpj_det": (192, 8e6),
                       "grad": (192, 8e6), "pj4": (128, 2e7), "bpj4": (128, 2e7)}.get(op, (256, 3e7))
    n = _log(rng, 16, top_n)
    if rng.random() < 0.3:                         # an anisotropic cube
        n = tuple(max(9, int(n * rng.uniform(0.6, 1.0))) for _ in range(3))
    N = (_log(rng, 24, 512),) * 2
    if rng.random() < 0.4:                         # a non-square image
        N = (N[0], max(17, int(N[0] * rng.uniform(0.6, 1.0))))
    T = max(3, min(_log(rng, 6, 400), int(top_rays / (N[0] * N[1]))))
    if N[0] * N[1] * T > top_rays:
        N, T = (181, 203), 4
    if op in ("pj4", "bpj4"):
        f = rng.randint(2, 12)
        T = max(f, T - T % f)
        kw["frames"] = f
    if op in ("pj", "bpj", "grad") and rng.random() < 0.3:
        kw["mask"] = True
    return _case(None, op, n, T, N, **kw)


# ---------------------------------------------------------------------------
# geometry

def _cube_header(n):
    h = {"SIMPLE": True, "BITPIX": -32, "NAXIS": 3}
    for k in range(3):
        h["NAXIS%d" % (k + 1)] = n[k]
        h["CRPIX%d" % (k + 1)] = n[k] / 2.0
        h["CDELT%d" % (k + 1)] = 3.0 / n[k]
        h["CRVAL%d" % (k + 1)] = 0.0
    return h


def _view_headers(c):
    d = c["d"]
    step = 2.0 * math.atan(1.6 / d) / max(c["N1"], c["N2"])
    out = []
    for lon in np.linspace(c["lon0"], c["lon1"], c["T"]):
        lat, rol = c["lat"] * math.cos(lon), c["rol"]
        out.append({"SIMPLE": True, "BITPIX": -32, "NAXIS": 2, "NAXIS1": c["N1"], "NAXIS2": c["N2"],
                    "CRPIX1": c["N1"] / 2.0, "CRPIX2": c["N2"] / 2.0, "CDELT1": step, "CDELT2": step,
                    "CRVAL1": 0.0, "CRVAL2": 0.0, "LON": float(lon), "LAT": lat, "ROL": rol, "D": d,
                    "M1": d * math.cos(lat) * math.cos(lon), "M2": d * math.cos(lat) * math.sin(lon),
                    "M3": d * math.sin(lat)})
    return out


def _frames(c):
    return np.arange(c["T"]) * c["frames"] // c["T"]


def _job_cases(c):
    """The jobs of a pack: edges and sides of the uneven mix."""
    rng = np.random.default_rng(c["jseed"])
    out = []
    for _ in range(c["jobs"]):
        n, N = int(rng.choice(EDGES)), int(rng.choice(SIDES))
        T = int(rng.integers(max(3, c["T"] // 4), c["T"] + 1))
        out.append(_case(None, "pj", n, T, N, d=float(rng.uniform(150.0, 230.0)), lon0=c["lon0"],
                         lon1=c["lon0"] + float(rng.uniform(3.0, 6.0))))
    return out


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _phantom(n, g, dtype=torch.float32):
    """A radial electron-density shell with eight Gaussian blobs (amplitudes of
    order one): the density the reconstructions look for."""
    ax = [(torch.arange(m, device="cuda", dtype=torch.float32) + 0.5) * (3.0 / m) - 1.5 for m in n]
    X, Y, Z = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    r = torch.sqrt(X * X + Y * Y + Z * Z)
    shell = (r > 1.05) & (r < 1.5)
    out = torch.exp(-(r - 1.0) / 0.1)
    v = torch.randn(8, 3, generator=g, device="cuda")
    v = v / v.norm(dim=1, keepdim=True) * (1.1 + 0.3 * torch.rand(8, 1, generator=g, device="cuda"))
    for k in range(8):
        q = (X - v[k, 0]) ** 2 + (Y - v[k, 1]) ** 2 + (Z - v[k, 2]) ** 2
        out = out + 0.3 * torch.exp(q * (-1.0 / (2 * 0.05 ** 2)))
    out = torch.where(shell, out, torch.zeros((), device="cuda"))
    return (out + 0.01 * torch.rand(tuple(n), generator=g, device="cuda")).to(dtype)


def _intensity(shape, g, dtype=torch.float32):
    """A positive image stack (views, rows, columns) with noise, seen as
    (rows, columns, views)."""
    n1, n2, T = shape
    i = torch.linspace(-1.6, 1.6, n1, device="cuda")[:, None]
    j = torch.linspace(-1.6, 1.6, n2, device="cuda")[None, :]
    prof = torch.exp(-(torch.sqrt(i * i + j * j) - 1.0).abs() / 0.4)
    y = prof * (0.6 + 0.4 * torch.rand(T, n1, n2, generator=g, device="cuda"))
    return y.to(dtype).permute(1, 2, 0)


def _mask(c, g):
    if not c["mask"]:
        return None
    i = torch.linspace(-1.6, 1.6, c["N1"], device="cuda")[:, None]
    j = torch.linspace(-1.6, 1.6, c["N2"], device="cuda")[None, :]
    out = ((i * i + j * j) < 0.5 ** 2)[:, :, None] | (torch.rand(c["N1"], c["N2"], c["T"], generator=g,
                                                                 device="cuda") < 0.02)
    return out.to(torch.uint8)


# ---------------------------------------------------------------------------
# what a program has in hand, and one pass

def prepare(case, seed):
    c, g = case, _gen(seed)
    op, n = c["op"], (c["n0"], c["n1"], c["n2"])
    obstacle = "sun" if c["sun"] else None
    shape = (c["N1"], c["N2"], c["T"])
    s = dict(case=c, op=op)
    if op == "packed":
        jobs = [batch.Job(_cube_header((j["n0"], j["n1"], j["n2"])), _view_headers(j)) for j in _job_cases(c)]
        s["pack"] = batch.PackedJobs(jobs, obstacle="sun", rows_per_warp=4)
        s["x"], s["z"] = s["pack"].new_cube(), s["pack"].new_cube()
        for k, j in enumerate(jobs):
            s["pack"].cube_view(s["x"], k).copy_(_phantom(j.cube_shape, g))
        return s
    ch, vh = _cube_header(n), _view_headers(c)
    m = _mask(c, g)
    if op == "dropin_pj":
        s.update(ch=ch, vh=vh, obstacle=obstacle, x=_phantom(n, g), y=torch.zeros(shape, device="cuda"))
        return s
    kw = dict(obstacle=obstacle, mask=m, dtype=np.float64 if op == "normal64" else np.float32)
    if op in ("pj4", "bpj4"):
        kw.update(frames=_frames(c), cube_shape=n + (c["frames"],))
    s["P"] = lo_wrapper.Siddon(vh, ch, deterministic=(op == "bpj_det"), **kw)
    if op in ("pj", "cg", "grad"):
        s["x"] = _phantom(n, g)
    elif op == "normal64":
        s["x"] = _phantom(n, g, torch.float64)
    elif op == "pj4":
        x = s["P"].new_cube()
        for f in range(c["frames"]):
            x[..., f] = _phantom(n, g)
        s["x"] = x
    else:
        s["y"] = _intensity(shape, g)
    if op == "grad":
        s["y0"] = _intensity(shape, g)
    if op == "cg":
        s["A"] = cg.NormalOperator(s["P"], lam=CG_LAM)
        s["b"] = s["P"].backproject(s["P"].project(s["x"]))
    return s


def run(s):
    op = s["op"]
    if op == "dropin_pj":
        s["y"].zero_()
        return tg.projector(s["y"], s["x"], obstacle=s["obstacle"], data_header=s["vh"], cube_header=s["ch"])
    if op == "packed":
        y = s["pack"].project(s["x"])
        return [y, s["pack"].backproject(s["z"])]
    P = s["P"]
    if op in ("pj", "pj4"):
        return P.project(s["x"])
    if op in ("bpj", "bpj4", "bpj_det"):
        return P.backproject(s["y"])
    if op == "normal64":
        y = P.project(s["x"])
        return [y, P.backproject(y)]
    if op == "grad":
        x = s["x"].detach().requires_grad_(True)
        y = autograd.project(x, P)
        loss = 0.5 * ((y - s["y0"]) ** 2).sum()
        loss.backward()
        return [y.detach(), x.grad]
    r = cg.cg(s["A"], s["b"], maxiter=CG_ITERS)
    return [r.x, np.asarray(r.residuals)]


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _crossings(c):
    """Rays and voxel crossings of a geometry, estimated: the cube fills
    3 / 3.2 of the wider image side, a ray that meets it crosses about 1.2
    planes of an in-plane axis per voxel of depth, and the sphere of radius
    one hides the back half of the rays that hit it."""
    rays = c["T"] * c["N1"] * c["N2"]
    hit = rays * 0.94 * 0.97
    depth = 1.25 * (c["n0"] + c["n1"]) / 2.0
    return rays, hit * depth * (0.7 if c["sun"] else 1.0)


def work(case):
    c = case
    if c["op"] == "packed":
        w = [work(dict(j, op="pj")) for j in _job_cases(c)]
        return {"bytes": 2 * sum(v["bytes"] for v in w), "flops": 2 * sum(v["flops"] for v in w)}
    rays, cross = _crossings(c)
    vox = c["n0"] * c["n1"] * c["n2"] * (c["frames"] if c["op"] in ("pj4", "bpj4") else 1)
    size = 8 if c["op"] == "normal64" else 4
    once = dict(bytes=size * (vox + rays) + (rays if c["mask"] else 0), flops=2 * cross)
    times = {"normal64": 2, "grad": 2, "cg": 2 * CG_ITERS}.get(c["op"], 1)
    return {k: times * v for k, v in once.items()}


# ---------------------------------------------------------------------------
# the same results in 64 bits: every ray is cut at the planes of its dominant
# axis; inside such a slab each other axis has at most one plane to cross, so
# a slab holds at most three pieces, each in the voxel of its midpoint

def _directions(c, t0, t1):
    hs = _view_headers(c)[t0:t1]
    dev = dict(device="cuda", dtype=torch.float64)
    gam = (torch.arange(c["N1"], **dev) - hs[0]["CRPIX1"] + 1) * hs[0]["CDELT1"]
    lam = (torch.arange(c["N2"], **dev) - hs[0]["CRPIX2"] + 1) * hs[0]["CDELT2"]
    cl, sl = torch.cos(lam)[None, :, None], torch.sin(lam)[None, :, None]
    cg_, sg = torch.cos(gam)[:, None, None], torch.sin(gam)[:, None, None]
    u, M = [], []
    lon = torch.tensor([h["LON"] for h in hs], **dev)
    lat = torch.tensor([h["LAT"] for h in hs], **dev)
    rol = torch.tensor([h["ROL"] for h in hs], **dev)
    a, b, e, f, p, q = lon.cos(), lon.sin(), lat.cos(), lat.sin(), rol.cos(), rol.sin()
    R = [[-a * e, -b * p - a * f * q, b * q - a * f * p],
         [-b * e, a * p - b * f * q, -a * q - b * f * p],
         [-f, e * q, e * p]]
    for k in range(3):
        v = R[k][0] * (cl * cg_) + R[k][1] * (cl * sg) + R[k][2] * (sl + 0 * cg_)
        u.append(torch.where(v.abs() < 1e-14, torch.zeros_like(v), v).reshape(-1))
        mk = torch.tensor([h["M%d" % (k + 1)] for h in hs], **dev)
        M.append(mk.expand(c["N1"], c["N2"], t1 - t0).reshape(-1))
    return torch.stack(u), torch.stack(M)


def _pieces(c, u, M, fbase):
    """(ray index, voxel index, length) of every piece, slab by slab."""
    n = torch.tensor([c["n0"], c["n1"], c["n2"]], device="cuda", dtype=torch.float64)[:, None]
    cd = 3.0 / n
    lo3 = -(n / 2.0) * cd
    hi3 = lo3 + cd * n
    zero = u == 0
    us = torch.where(zero, torch.ones_like(u), u)
    a1, an = (lo3 - M) / us, (hi3 - M) / us
    big = 1e5
    amin = torch.where(zero, torch.full_like(u, -big), torch.minimum(a1, an)).amax(0)
    amax = torch.where(zero, torch.full_like(u, big), torch.maximum(a1, an)).amin(0)
    flat = ((M - lo3) / cd).floor()
    ok = (amin < amax) & ~(zero & ((flat < 0) | (flat >= n))).any(0)
    rays = ok.nonzero().reshape(-1)
    if not rays.numel():
        return
    u, M, us, zero, flat, amin, amax, fbase = (v[..., rays] for v in (u, M, us, zero, flat, amin, amax, fbase))
    stride = torch.tensor([c["n1"] * c["n2"], c["n2"], 1], device="cuda", dtype=torch.float64)[:, None]
    k = (u.abs() / cd).argmax(0)
    order = torch.stack([k, (k + 1) % 3, (k + 2) % 3])
    take = lambda v: torch.gather(v.expand(3, rays.numel()), 0, order)   # noqa: E731
    u, us, M, zero, flat = take(u), take(us), take(M), take(zero), take(flat)
    n, cd, lo3, stride = take(n), take(cd), take(lo3), take(stride)
    org, slope = (M - lo3) / cd, u / cd                # position in voxels: org + t slope
    inv = cd / us
    sc = -(M * u).sum(0)
    gap = (M * M).sum(0) - sc * sc - 1.0               # |r(t)|^2 - 1 = (t - sc)^2 + gap
    alive = torch.ones_like(sc, dtype=torch.bool)
    up = u[0] > 0
    nk = int(n[0].max())

    def index(a, t):                                   # voxel of axis a at parameter t
        p = torch.addcmul(org[a], t, slope[a]).floor_()
        if a:
            p = torch.where(zero[a], flat[a], p)
        return torch.minimum(p.clamp_(min=0), n[a] - 1)

    def plane(a, e, f):                                # parameter where axis a crosses in [e, f], or f
        q = torch.maximum(torch.addcmul(org[a], e, slope[a]).floor_(), torch.addcmul(org[a], f, slope[a]).floor_())
        return torch.where(zero[a], f, torch.minimum(torch.maximum((q - org[a]) * inv[a], e), f))

    for s in range(nk):
        q0 = torch.where(up, torch.full_like(sc, float(s)), n[0] - s)
        q1 = torch.where(up, q0 + 1, q0 - 1)
        e = torch.maximum((q0 - org[0]) * inv[0], amin)
        f = torch.minimum((q1 - org[0]) * inv[0], amax)
        here = (f > e) & (s < n[0])
        f = torch.maximum(e, f)
        ia = torch.where(up, q0, q1) * stride[0] + fbase
        ta, tb = plane(1, e, f), plane(2, e, f)
        cut = (e, torch.minimum(ta, tb), torch.maximum(ta, tb), f)
        for p in range(3):
            x0, x1 = cut[p], cut[p + 1]
            L = x1 - x0
            if c["sun"]:
                alive &= ~(here & (L > 0)) | ((x0 - sc) ** 2 + gap > 0)
            mid = (x0 + x1) * 0.5
            vox = ia + index(1, mid) * stride[1] + index(2, mid) * stride[2]
            L = L * (here & alive)
            yield rays, torch.where(L > 0, vox, torch.zeros_like(vox)).long(), L


def _frame_base(c, t0, t1):
    f = torch.from_numpy(_frames(c)[t0:t1] * (c["n0"] * c["n1"] * c["n2"])).cuda().double()
    return f.expand(c["N1"], c["N2"], t1 - t0).reshape(-1)


def _chunks(c):
    step = max(1, (1 << 20) // (c["N1"] * c["N2"]))
    for t0 in range(0, c["T"], step):
        yield t0, min(c["T"], t0 + step)


def _exact_pj(c, x, mask=None):
    """x: float64 cube, frames outermost when it has them -> (N1, N2, T)."""
    x = x.reshape(-1)
    out = torch.zeros(c["N1"], c["N2"], c["T"], device="cuda", dtype=torch.float64)
    for t0, t1 in _chunks(c):
        u, M = _directions(c, t0, t1)
        acc = torch.zeros(u.shape[1], device="cuda", dtype=torch.float64)
        part = None
        for rays, vox, L in _pieces(c, u, M, _frame_base(c, t0, t1)):
            part = torch.zeros_like(L) if part is None else part
            part.addcmul_(L, x[vox])
        if part is not None:
            acc[rays] = part
        out[:, :, t0:t1] = acc.view(c["N1"], c["N2"], t1 - t0)
    return out if mask is None else torch.where(mask != 0, torch.zeros_like(out), out)


def _exact_bpj(c, y, mask=None):
    """y: (N1, N2, T) -> float64 cube (frames, n0, n1, n2)."""
    y = y.double()
    if mask is not None:
        y = torch.where(mask != 0, torch.zeros_like(y), y)
    out = torch.zeros(c["frames"] * c["n0"] * c["n1"] * c["n2"], device="cuda", dtype=torch.float64)
    for t0, t1 in _chunks(c):
        u, M = _directions(c, t0, t1)
        yc = y[:, :, t0:t1].reshape(-1)
        yr = None
        for rays, vox, L in _pieces(c, u, M, _frame_base(c, t0, t1)):
            yr = yc[rays] if yr is None else yr
            out.index_add_(0, vox, L * yr)
    return out.view(c["frames"], c["n0"], c["n1"], c["n2"])


def exact(case, seed):
    c = case
    if c["op"] != "packed" and c["T"] * c["N1"] * c["N2"] * max(c["n0"], c["n1"], c["n2"]) > 1.4e10:
        return None                                    # the largest orbits take too long in 64 bits
    s = prepare(c, seed)
    op = c["op"]
    m = s["P"].mask if "P" in s else None
    if op == "packed":
        ys, zs = [], []
        pack = s["pack"]
        for k, j in enumerate(_job_cases(c)):
            y = _exact_pj(j, pack.cube_view(s["x"], k).double())
            ys.append(y.permute(2, 0, 1).reshape(-1))
            zs.append(_exact_bpj(j, y).reshape(-1))
        return [torch.cat(ys), torch.cat(zs)]
    if op in ("dropin_pj", "pj"):
        return _exact_pj(c, s["x"].double(), m)
    if op == "pj4":
        return _exact_pj(c, s["x"].permute(3, 0, 1, 2).double(), m)
    if op in ("bpj", "bpj_det"):
        return _exact_bpj(c, s["y"], m)[0]
    if op == "bpj4":
        return _exact_bpj(c, s["y"], m).permute(1, 2, 3, 0)
    if op == "normal64":
        y = _exact_pj(c, s["x"])
        return [y, _exact_bpj(c, y)[0]]
    if op == "grad":
        y = _exact_pj(c, s["x"].double(), m)
        return [y, _exact_bpj(c, y - s["y0"].double(), m)[0]]
    A = lambda v: _exact_bpj(c, _exact_pj(c, v))[0] + CG_LAM * v      # noqa: E731
    b = s["b"].double()
    x, r, p = torch.zeros_like(b), b.clone(), b.clone()
    rr, bb = float((r * r).sum()), float((b * b).sum())
    hist = [1.0]
    for _ in range(CG_ITERS):
        q = A(p)
        alpha = rr / float((p * q).sum())
        x, r = x + alpha * p, r - alpha * q
        new = float((r * r).sum())
        p, rr = r + (new / rr) * p, new
        hist.append(math.sqrt(rr / bb))
    return [x, np.asarray(hist)]
