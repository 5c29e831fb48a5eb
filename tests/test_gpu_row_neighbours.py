"""A ray of the row walk (csrc/siddon_rows.cuh) has the same bits whatever is
traced beside it: with its neighbours masked, alone, and in the 8- and
16-column tiles of lanes along image axis 0.

Cubes above and below the observer's plane: rays enter them through a face of
cube axis 2 at different row segments (chords of up to 90 segments); and a cube
around it, entered through the other faces."""
import numpy as np
import pytest

from tomograpy_gb300 import batch, lo_wrapper, siddon
from tomograpy_gb300 import headers as H

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

N, T = (24, 64), 4


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def _geometry(z):
    ch = H.centered_cubic_map_header([3.0, 3.0, 3.0], (48, 48, 48), dtype=np.float32)
    if abs(z) > 1.0:                               # the cube's face at z, the cube behind it
        ch["CRPIX3"] = -24.0 if z > 0 else 72.0
        H.map_borders(ch)
    vh = []
    for lon in np.linspace(0.13, 5.9, T):
        h = H.centered_image_header(1e-3, N, dtype=np.float32)
        h.update({"CDELT1": 3.2 / 215.0 / N[0], "CDELT2": 5e-4 / 215.0, "CRVAL2": float(np.arctan(z / 215.0)),
                  "LON": float(lon), "LAT": 0.0, "ROL": 0.0, "D": 215.0, "M1": 215.0 * np.cos(lon),
                  "M2": 215.0 * np.sin(lon), "M3": 0.0})
        H.header_rotation_matrix(h)
        vh.append(h)
    return ch, vh


@pytest.mark.parametrize("obstacle", [None, "sun"])
@pytest.mark.parametrize("z", [1.5, -1.498, 0.3])
def test_projection_does_not_depend_on_the_rays_beside(z, obstacle):
    ch, vh = _geometry(z)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand(48, 48, 48, generator=g, device="cuda") + 0.1
    want = lo_wrapper.siddon_lo(vh, ch, obstacle=obstacle, dtype=np.float32).project(x)
    assert bool((want > 0).any())
    tab, mh = siddon.upload_views(vh), siddon.pack_map_header(ch)
    for seed in range(3):
        m = (torch.rand(N + (T,), generator=g, device="cuda") < 0.5 + 0.2 * seed).to(torch.uint8)
        got = torch.zeros(N + (T,), device="cuda")
        siddon.run_device("pj", got, x, tab, mh, T, m, obstacle)
        assert torch.equal(got, torch.where(m != 0, torch.zeros_like(want), want))
    for j in range(0, N[1], 7):
        got = torch.zeros(N + (T,), device="cuda")
        siddon.run_device("pj", got, x, tab, mh, T, None, obstacle, ray=(11, j, 2))
        assert float(got[11, j, 2]) == float(want[11, j, 2])
    job = batch.Job(ch, vh)
    for sched in ((1, 0, 0), (2, 0, 0), (4, 0, 0), (1, 1, 0)):
        pack = batch.PackedJobs([job], obstacle=obstacle, schedule=sched)
        flat = pack.new_cube()
        pack.cube_view(flat, 0).copy_(x)
        pack.project(flat)
        assert torch.equal(pack.data_view(pack.data, 0), want), sched
