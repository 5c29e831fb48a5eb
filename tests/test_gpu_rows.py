"""The row walk (csrc/siddon_rows.cuh: views whose lambda axis runs along cube
axis 2) at the sizes where it can go wrong, against the float64 oracle and
against the general walk.

A latitude of 1e-12 rad makes R[0][2], R[1][2] non-zero, so the same view takes
the general walk; the rays move by 215 * 1e-12 radii, far below float32.  Both
walks are within the image / cube tolerances of the float64 result, so they
are within twice those of each other."""
import numpy as np
import pytest

from helpers import CUBE_TOL, IMG_TOL, cube_errors, degenerate_rays, image_errors
from tomograpy_gb300 import headers as H
from tomograpy_gb300 import lo_wrapper, siddon, synthetic
from tomograpy_gb300.infoarray import InfoArray

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def _cube_header(n):
    return H.centered_cubic_map_header([3.0 * m / max(n) for m in n], n, dtype=np.float32)


def _views(T, N, d, lat=0.0, fov=1.6, off=0.0):
    lons = np.linspace(0.13, 5.9, T)
    step = 2.0 * np.arctan(fov / d) / max(N)
    out = []
    for lon in lons:
        h = H.centered_image_header(step, N, dtype=np.float32)
        h.update({"CDELT1": step, "CDELT2": step, "CRVAL2": off * step, "LON": float(lon), "LAT": lat, "ROL": 0.0,
                  "D": float(d), "M1": d * np.cos(lat) * np.cos(lon), "M2": d * np.cos(lat) * np.sin(lon),
                  "M3": d * np.sin(lat)})
        H.header_rotation_matrix(h)
        out.append(h)
    return out


# cube, image (rows, columns), views, observer distance, half field of view,
# column offset: one voxel; fewer columns than a warp; one more than a tile's
# blocks; windows of 32 row segments with a remainder; long thin cubes; images
# much coarser and much finer than the voxels (several planes in one segment
# group, many rays per voxel); rays off to one side (entry and exit through
# faces of axis 2); an observer so near that rows fall back; one inside
GEOMETRIES = [((1, 1, 1), (5, 7), 3, 215.0, 1.6, 0.0), ((9, 14, 11), (33, 31), 4, 215.0, 1.6, 0.0),
              ((33, 31, 40), (9, 129), 4, 180.0, 1.6, 0.3), ((64, 65, 63), (40, 40), 5, 215.0, 1.6, 0.0),
              ((130, 7, 64), (64, 33), 4, 150.0, 1.6, 0.0), ((24, 24, 192), (17, 65), 3, 200.0, 1.6, 0.0),
              ((16, 16, 16), (70, 260), 3, 215.0, 1.6, 0.0), ((48, 48, 48), (60, 60), 4, 215.0, 1.2, 55.0),
              ((40, 40, 40), (32, 48), 5, 6.0, 1.6, 0.0), ((20, 20, 20), (24, 24), 4, 1.2, 3.0, 0.0)]


@pytest.mark.parametrize("obstacle", [None, "sun"])
@pytest.mark.parametrize("geo", GEOMETRIES, ids=lambda g: "x".join(map(str, g[0])))
def test_row_walk_matches_oracle(geo, obstacle):
    import oracle
    n, N, T, d, fov, off = geo
    ch, vh = _cube_header(n), _views(T, N, d, fov=fov, off=off)
    rng = np.random.default_rng(sum(n))
    x = (0.2 + rng.random(n)).astype(np.float32)
    y = (0.2 + rng.random(N + (T,))).astype(np.float32)
    deg = degenerate_rays(vh, *N)
    y[deg] = 0.0
    op = lo_wrapper.siddon_lo(vh, ch, obstacle=obstacle, dtype=np.float32)
    ref = InfoArray(shape=N + (T,), header=[dict(h) for h in vh], dtype=np.float64)
    oracle.projector(ref, InfoArray(data=x.astype(np.float64), header=dict(ch)), obstacle=obstacle)
    rel, norm = image_errors(op.project(torch.from_numpy(x)).cpu().numpy(), ref, exclude=deg)
    assert rel <= IMG_TOL and norm <= IMG_TOL, (rel, norm)
    cref = InfoArray(shape=n, header=dict(ch), dtype=np.float64)
    oracle.backprojector(InfoArray(data=y.astype(np.float64), header=[dict(h) for h in vh]), cref, obstacle=obstacle)
    rel, norm = cube_errors(op.backproject(torch.from_numpy(y)).cpu().numpy(), cref, float(y.max()),
                            min(ch["CDELT%d" % (k + 1)] for k in range(3)))
    assert rel <= CUBE_TOL and norm <= CUBE_TOL, (rel, norm)
    det = lo_wrapper.siddon_lo(vh, ch, obstacle=obstacle, dtype=np.float32, deterministic=True)
    rel, norm = cube_errors(det.backproject(torch.from_numpy(y)).cpu().numpy(), cref, float(y.max()),
                            min(ch["CDELT%d" % (k + 1)] for k in range(3)))
    assert rel <= CUBE_TOL and norm <= CUBE_TOL, (rel, norm)


@pytest.mark.parametrize("mask", [None, torch.uint8, torch.float32, torch.float64])
@pytest.mark.parametrize("order", [(0, 1, 2), (2, 1, 0), (1, 0, 2)])
@pytest.mark.parametrize("frames", [None, (0, 2, 2, 1, 0)])
def test_row_walk_matches_general_walk(order, mask, frames):
    """Cube axis orders, data layouts, masks, frame tables, overwriting and
    single views, each through both walks."""
    n, N, T, d = (21, 34, 26), (19, 45), 5, 215.0
    ch = _cube_header(n)
    g = torch.Generator(device="cuda").manual_seed(5)
    shape = n + ((3,) if frames else ())
    perm = list(order) + ([3] if frames else [])
    store = torch.rand([shape[p] for p in perm], generator=g, device="cuda") + 0.1
    x = store.permute([perm.index(k) for k in range(len(perm))])
    y = torch.rand((T,) + N, generator=g, device="cuda").permute(1, 2, 0)
    m = None if mask is None else (torch.rand(N + (T,), generator=g, device="cuda") < 0.2).to(mask)
    both = []
    for lat in (0.0, 1e-12):
        vh = _views(T, N, d, lat=lat)
        tab, mh = siddon.upload_views(vh, frames), siddon.pack_map_header(ch)
        fwd, bwd = ("pjt", "bpjt") if frames else ("pj", "bpj")
        img = torch.zeros(N + (T,), device="cuda")
        siddon.run_device(fwd, img, x, tab, mh, T, m, "sun")
        ovw = torch.full(N + (T,), 7.0, device="cuda")
        siddon.run_device(fwd, ovw, x, tab, mh, T, m, "sun", overwrite=True)
        one = torch.zeros(N + (T,), device="cuda")
        siddon.run_device(fwd, one, x, tab, mh, T, m, "sun", view=3)
        assert torch.equal(ovw, img) and torch.equal(one[..., 3], img[..., 3])
        cube = torch.zeros_like(store).permute([perm.index(k) for k in range(len(perm))])
        siddon.run_device(bwd, y, cube, tab, mh, T, m, "sun")
        both.append((img.cpu().numpy(), cube.cpu().numpy()))
    (ia, ca), (ib, cb) = both
    rel, norm = image_errors(ia, ib)
    assert rel <= 2 * IMG_TOL and norm <= 2 * IMG_TOL, (rel, norm)
    rel, norm = cube_errors(ca, cb, float(y.max()), ch["CDELT1"])
    assert rel <= 2 * CUBE_TOL and norm <= 2 * CUBE_TOL, (rel, norm)


def test_row_walk_keeps_non_finite_voxels_to_their_rays():
    """An infinite voxel reaches the rays that pass through it, and no other."""
    ch, vh = synthetic.make_geometry(dict(n=32, T=3, N=64, d=215.0, lon_range=(0.2, 2.9)))
    op = lo_wrapper.siddon_lo(vh, ch, dtype=np.float32)
    x = torch.zeros(32, 32, 32, device="cuda")
    x[14, 17, 21] = 1.0
    chord = op.project(x)
    x[14, 17, 21] = float("inf")
    y = op.project(x)
    through = chord > 1e-5
    assert through.any() and torch.isinf(y[through]).all()
    assert (y[chord == 0] == 0).all()


def test_row_walk_makes_no_nan_of_corners():
    """Rays along a diagonal of the cells cross two plane families at once; the
    cells that only share the corner are not passed, and 0 * inf is not formed."""
    n, N = 16, 32
    ch = _cube_header((n, n, n))
    vh = [h for lon in (np.pi / 4, 3 * np.pi / 4) for h in synthetic.view_headers(1, N, lons=[lon])]
    op = lo_wrapper.siddon_lo(vh, ch, dtype=np.float32)
    i = torch.arange(n, device="cuda")
    x = torch.ones(n, n, n, device="cuda")
    x[(i[:, None] - i[None, :]).abs() == 1] = float("inf")
    assert not torch.isnan(op.project(x)).any()
    y = torch.zeros(N, N, 2, device="cuda")
    y[N // 2 - 1] = float("inf")
    assert not torch.isnan(op.backproject(y)).any()
