"""Row-walk views in packs whose lanes run along image axis 0: tiles of 8 and 16
columns share the rows of 32 columns between them (tile_body,
csrc/siddon_fast.cuh).  Images whose last 32 columns hold one to four tiles, and
rows that end inside a tile: every pixel is traced once, with the bits of the
single-job kernel; the backprojection against the oracle."""
import numpy as np
import pytest

from helpers import CUBE_TOL, cube_errors, degenerate_rays
from tomograpy_gb300 import batch, lo_wrapper
from tomograpy_gb300 import headers as H
from tomograpy_gb300.infoarray import InfoArray

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def _job(n, N, T=3):
    ch = H.centered_cubic_map_header([3.0, 3.0, 3.0], n, dtype=np.float32)
    step, vh = 2.0 * np.arctan(1.6 / 215.0) / max(N), []
    for lon in np.linspace(0.13, 5.9, T):
        h = H.centered_image_header(step, N, dtype=np.float32)
        h.update({"CDELT1": step, "CDELT2": step, "LON": float(lon), "LAT": 0.0, "ROL": 0.0, "D": 215.0,
                  "M1": 215.0 * np.cos(lon), "M2": 215.0 * np.sin(lon), "M3": 0.0})
        H.header_rotation_matrix(h)
        vh.append(h)
    return ch, vh


SIZES = [(5, 7), (33, 8), (31, 9), (40, 17), (64, 33), (37, 40), (35, 56), (70, 57), (32, 64)]


@pytest.mark.parametrize("rows", [1, 2, 4])
def test_columns_of_gamma_lanes(rows):
    import oracle
    n = (12, 10, 14)
    geo = [_job(n, N) for N in SIZES]
    pack = batch.PackedJobs([batch.Job(ch, vh) for ch, vh in geo], obstacle="sun", schedule=(rows, 0, 0))
    rng = np.random.default_rng(rows)
    cubes = [(0.2 + rng.random(n)).astype(np.float32) for _ in geo]
    flat = pack.new_cube()
    for k, x in enumerate(cubes):
        pack.cube_view(flat, k).copy_(torch.from_numpy(x))
    pack.project(flat)
    for k, (ch, vh) in enumerate(geo):
        want = lo_wrapper.siddon_lo(vh, ch, obstacle="sun", dtype=np.float32).project(torch.from_numpy(cubes[k]).cuda())
        assert bool((want > 0).any())
        assert torch.equal(pack.data_view(pack.data, k), want), SIZES[k]
    ys = []
    for k, (ch, vh) in enumerate(geo):
        y = 0.2 + rng.random(SIZES[k] + (len(vh),))
        y[degenerate_rays(vh, *SIZES[k])] = 0.0
        ys.append(y.astype(np.float32))
        pack.data_view(pack.data, k).copy_(torch.from_numpy(ys[k]))
    pack.backproject(flat)
    for k, (ch, vh) in enumerate(geo):
        ref = InfoArray(shape=n, header=dict(ch), dtype=np.float64)
        oracle.backprojector(InfoArray(data=ys[k].astype(np.float64), header=[dict(h) for h in vh]), ref, obstacle="sun")
        rel, norm = cube_errors(pack.cube_view(flat, k).cpu().numpy(), ref, float(ys[k].max()), ch["CDELT1"])
        assert rel <= CUBE_TOL and norm <= CUBE_TOL, (SIZES[k], rel, norm)
