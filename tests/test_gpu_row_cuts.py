"""Rays of the row walk (csrc/siddon_rows.cuh) at planes of cube axis 2: the
parts of the row segment that holds the plane.

An observer at 215 radii on axis 0; every ray crosses plane z = 0.9375 of the
cube a distance eps behind the cube's middle plane x = 0, eps in steps of 1e-3
radii along the image row.  The voxel between the two planes holds a path of
eps, nothing else of the ray counts.

Tolerance: near the chord's middle, where the walk's parameters have their
origin, crossings are exact to 1e-11 radii (double-float set-up) plus 2^-24 of
their small distance from it; the length, 1 / cos(lambda) and the product round
at 2^-24 each: below 1e-6 of eps >= 1e-3 with room to spare."""
import numpy as np
import pytest

from tomograpy_gb300 import headers as H
from tomograpy_gb300 import lo_wrapper
from tomograpy_gb300.infoarray import InfoArray

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

N = (2, 64)


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def _geometry(n):
    d, z = 215.0, 0.9375
    ch = H.centered_cubic_map_header([3.0, 3.0, 3.0], n, dtype=np.float32)
    h = H.centered_image_header(2e-4, N, dtype=np.float32)
    # columns at tan(lambda) = z / (d + eps): eps = 1e-3 (63 - j) behind x = 0
    lam = np.arctan(z / (d + 1e-3 * np.array([63.0, 0.0])))
    step = (lam[1] - lam[0]) / (N[1] - 1)
    h.update({"CDELT1": 2e-4, "CRVAL1": 3e-4, "CDELT2": step, "CRPIX2": 1.0, "CRVAL2": lam[0], "LON": 0.0,
              "LAT": 0.0, "ROL": 0.0, "D": d, "M1": d, "M2": 0.0, "M3": 0.0})
    H.header_rotation_matrix(h)
    return ch, [h]


def _oracle(ch, vh, x):
    import oracle
    ref = InfoArray(shape=N + (1,), header=[dict(h) for h in vh], dtype=np.float64)
    H.map_borders(ch)
    oracle.projector(ref, InfoArray(data=x.astype(np.float64), header=dict(ch)))
    return np.asarray(ref)


def _voxel(ch, n):
    """The voxel behind x = 0 and below z = 0.9375, at the rows' y of 0.04 to 0.09."""
    i = [n[0] // 2 - 1, int((0.06 + 1.5) / 3.0 * n[1]), int(round((0.9375 + 1.5) / 3.0 * n[2])) - 1]
    return tuple(i)


# planes of axis 2 so far apart that this one is the ray's first
@pytest.mark.parametrize("n", [(16, 16, 16), (32, 4, 16)])
def test_parts_of_a_cut_segment(n):
    ch, vh = _geometry(n)
    x = np.zeros(n, np.float32)
    v = _voxel(ch, n)
    x[v] = 1.0
    ref = _oracle(ch, vh, x)
    eps = ref[0, :, 0]
    long = (eps > 9e-4) & (eps < 0.05)
    assert long.sum() > 40
    op = lo_wrapper.siddon_lo(vh, ch, dtype=np.float32)
    y = op.project(torch.from_numpy(x)).cpu().numpy().astype(np.float64)
    err = np.abs(y - ref)[:, long] / ref[:, long]
    assert err.max() <= 1e-6, err.max()
    # the same parts backprojected, one ray at a time: nothing negative, nothing beside its path
    for det in (False, True):
        op = lo_wrapper.siddon_lo(vh, ch, dtype=np.float32, deterministic=det)
        for j in np.flatnonzero(long)[::9]:
            w = torch.zeros(N + (1,), device="cuda")
            w[0, int(j)] = 1.0
            c = op.backproject(w).cpu().numpy()
            assert c.min() >= 0.0
            # a deterministic sum rounds to a fixed point of far below 2^-30
            assert abs(float(c[v]) - eps[j]) <= 1e-6 * eps[j], (det, j, c[v], eps[j])


def test_cut_segment_does_not_overflow():
    """A voxel so large that the whole segment's product is beyond float32, of
    which a ray passes a part that is not."""
    import oracle
    n = (8, 8, 8)
    ch = H.centered_cubic_map_header([40.0, 40.0, 40.0], n, dtype=np.float32)
    h = H.centered_image_header(2e-4, (2, 256), dtype=np.float32)
    h.update({"CDELT1": 2e-4, "CRVAL1": 3e-4, "CDELT2": 2e-6, "CRVAL2": float(np.arctan(15.0 / 215.0)), "LON": 0.0,
              "LAT": 0.0, "ROL": 0.0, "D": 215.0, "M1": 215.0, "M2": 0.0, "M3": 0.0})
    H.header_rotation_matrix(h)
    H.map_borders(ch)
    x = np.zeros(n, np.float64)
    x[3, 4, 6] = 1e38
    ref = InfoArray(shape=(2, 256, 1), header=[dict(h)], dtype=np.float64)
    oracle.projector(ref, InfoArray(data=x, header=dict(ch)))
    ref = np.asarray(ref)
    small = ref > 1e36
    assert small.sum() > 100 and ref.max() < 1e38
    y = lo_wrapper.siddon_lo([h], ch, dtype=np.float32).project(torch.from_numpy(x.astype(np.float32))).cpu().numpy()
    assert np.isfinite(y[small]).all()
    assert (np.abs(y[small] - ref[small]) <= 1e-5 * ref[small] + 1e33).all()


@pytest.mark.parametrize("lon", [np.pi / 4, 3 * np.pi / 4, -np.pi / 4])
def test_stop_at_a_corner_reads_nothing_behind_it(lon):
    """Rays along a diagonal of the cells that the sphere stops where they cross
    two plane families at once: no voxel inside the sphere, which no ray
    enters, is read or written."""
    n, rows = 16, 32
    ch = H.centered_cubic_map_header([3.0, 3.0, 3.0], (n, n, n), dtype=np.float32)
    h = H.centered_image_header(3.2 / 215.0, (rows, rows), dtype=np.float32)
    h.update({"CRPIX1": rows / 2.0, "CRPIX2": rows / 2.0, "LON": lon, "LAT": 0.0, "ROL": 0.0, "D": 215.0,
              "M1": 215.0 * np.cos(lon), "M2": 215.0 * np.sin(lon), "M3": 0.0})
    H.header_rotation_matrix(h)
    edge = np.abs(np.arange(n + 1) * 3.0 / n - 1.5)
    far = np.maximum(edge[1:], edge[:-1]) ** 2
    inside = torch.from_numpy(far[:, None, None] + far[None, :, None] + far[None, None, :] < 1.0).cuda()
    assert int(inside.sum()) > 100
    x = torch.where(inside, float("nan"), 1.0).float()
    for det in (False, True):
        op = lo_wrapper.siddon_lo([h], ch, obstacle="sun", dtype=np.float32, deterministic=det)
        assert bool(torch.isfinite(op.project(x)).all())
        y = torch.ones(rows, rows, 1, device="cuda")
        if not det:
            y[rows // 2 - 1] = float("inf")
        assert bool((op.backproject(y)[inside] == 0).all())


@pytest.mark.parametrize("n", [(16, 16, 1024), (32, 4, 1024)])
def test_parts_behind_earlier_planes(n):
    """The same voxel where the ray has crossed two planes of axis 2 before
    this one: its crossing is as exact as the first."""
    test_parts_of_a_cut_segment(n)
