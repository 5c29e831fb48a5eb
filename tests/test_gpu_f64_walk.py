"""The float64 walk (csrc/siddon_ref.cu) against the float64 oracle where its
short cuts change over: observers inside the cube (negative parameters), near
it and so far that the obstacle is tested at every voxel; rows that do not
fill a CTA; an image tall enough for eight rows per CTA.  Tolerance: the
float64 path's 1e-12 normwise."""
import numpy as np
import pytest

from helpers import degenerate_rays, image_errors
from tomograpy_gb300 import headers as H
from tomograpy_gb300 import lo_wrapper, synthetic
from tomograpy_gb300.infoarray import InfoArray

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def _views(T, N, d, lat):
    step = 2.0 * np.arctan(1.6 / d) / max(N)
    out = []
    for lon in np.linspace(0.17, 5.1, T):
        h = H.centered_image_header(step, N, dtype=np.float64)
        h.update({"CDELT1": step, "CDELT2": step, "LON": float(lon), "LAT": lat, "ROL": 0.2, "D": float(d),
                  "M1": d * np.cos(lat) * np.cos(lon), "M2": d * np.cos(lat) * np.sin(lon), "M3": d * np.sin(lat)})
        H.header_rotation_matrix(h)
        out.append(h)
    return out


@pytest.mark.parametrize("obstacle", [None, "sun"])
@pytest.mark.parametrize("n,N,T,d", [(20, (13, 45), 4, 1.2), (20, (13, 45), 4, 6.0), (33, (30, 31), 3, 215.0),
                                     (16, (9, 64), 3, 2e4), (1, (3, 5), 2, 215.0), (4, (4 * 65535 + 1, 1), 1, 215.0)])
def test_f64_matches_oracle(n, N, T, d, obstacle):
    import oracle
    ch, vh = synthetic.cube_header(n, dtype=np.float64), _views(T, N, d, 0.1)
    rng = np.random.default_rng(n)
    x = 0.2 + rng.random((n,) * 3)
    y = 0.2 + rng.random(N + (T,))
    deg = degenerate_rays(vh, *N)
    y[deg] = 0.0
    op = lo_wrapper.siddon_lo(vh, ch, obstacle=obstacle, dtype=np.float64)
    ref = InfoArray(shape=N + (T,), header=[dict(h) for h in vh], dtype=np.float64)
    oracle.projector(ref, InfoArray(data=x, header=dict(ch)), obstacle=obstacle)
    _, norm = image_errors(op.project(torch.from_numpy(x)).cpu().numpy(), ref, exclude=deg)
    assert norm <= 1e-12, norm
    cref = InfoArray(shape=(n,) * 3, header=dict(ch), dtype=np.float64)
    oracle.backprojector(InfoArray(data=y, header=[dict(h) for h in vh]), cref, obstacle=obstacle)
    _, norm = image_errors(op.backproject(torch.from_numpy(y)).cpu().numpy(), cref)
    assert norm <= 1e-12, norm


def test_f64_obstacle_with_rounded_rotation_matrices():
    """Headers that give the rotation matrix to nine decimals: directions up to
    1e-9 off unit length, which moves |r|^2 by 4e-5 at 215 radii, and rays
    within 5e-5 radii of the limb through planes 2e-3 radii apart.  Each ray
    stops at the voxel where the oracle stops."""
    import oracle
    n, N, T, d = (1500, 4, 4), (3, 96), 12, 215.0
    ch = H.centered_cubic_map_header([3.0, 3.0, 3.0], n, dtype=np.float64)
    vh = []
    for lon in np.linspace(-0.1, 0.1, T):
        h = H.centered_image_header(1e-5, N, dtype=np.float64)
        h.update({"CDELT1": 1e-5, "CDELT2": 1e-4 / d / N[1], "CRVAL2": float(np.arcsin(1.0 / d)), "LON": float(lon),
                  "LAT": 0.05, "ROL": 0.2, "D": d, "M1": d * np.cos(0.05) * np.cos(lon),
                  "M2": d * np.cos(0.05) * np.sin(lon), "M3": d * np.sin(0.05)})
        H.header_rotation_matrix(h)
        h.update({k: round(float(v), 9) for k, v in h.items() if k.startswith("R") and "_" in k})
        vh.append(h)
    x = 0.2 + np.random.default_rng(1).random(n)
    op = lo_wrapper.siddon_lo(vh, ch, obstacle="sun", dtype=np.float64)
    ref = InfoArray(shape=N + (T,), header=[dict(h) for h in vh], dtype=np.float64)
    oracle.projector(ref, InfoArray(data=x, header=dict(ch)), obstacle="sun")
    _, norm = image_errors(op.project(torch.from_numpy(x)).cpu().numpy(), ref)
    assert norm <= 1e-12, norm
