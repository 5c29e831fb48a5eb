"""Tiles of two, three and four 32-column blocks, which launches of many views
take (pick_tile, csrc/capi.cu: from 7296 tiles on), with a ragged last block and
a last tile of fewer blocks: the row walk and the general walk, masked and
overwriting, against the same 20 views in tiles of one block -- bit by bit, a
pixel does not depend on its tile -- which are checked against the oracle."""
import numpy as np
import pytest

from helpers import CUBE_TOL, IMG_TOL, cube_errors, degenerate_rays, image_errors
from tomograpy_gb300 import headers as H
from tomograpy_gb300 import siddon
from tomograpy_gb300.infoarray import InfoArray

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

FEW, TIMES, n = 20, 185, (9, 12, 10)


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def _views(N, lat):
    out = []
    step = 2.0 * np.arctan(1.6 / 215.0) / max(N)
    for lon in np.linspace(0.13, 5.9, FEW):
        h = H.centered_image_header(step, N, dtype=np.float32)
        h.update({"CDELT1": step, "CDELT2": step, "LON": float(lon), "LAT": lat, "ROL": 2.0 * lat, "D": 215.0,
                  "M1": 215.0 * np.cos(lat) * np.cos(lon), "M2": 215.0 * np.cos(lat) * np.sin(lon),
                  "M3": 215.0 * np.sin(lat)})
        H.header_rotation_matrix(h)
        out.append(h)
    return out


# columns: 2 blocks (1 and 32 columns in the last), 3, 4, and 4 + 1
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("lat", [0.0, 0.1])
@pytest.mark.parametrize("cols", [33, 64, 65, 97, 129])
def test_wide_tiles(cols, lat, masked):
    import oracle
    N = (35, cols)
    assert 2 * FEW * 5 < 7296 <= 2 * FEW * TIMES         # one block / all of them
    ch, vh = H.centered_cubic_map_header([3.0, 3.0, 3.0], n, dtype=np.float32), _views(N, lat)
    rng = np.random.default_rng(cols)
    x64, y64 = 0.2 + rng.random(n), 0.2 + rng.random(N + (FEW,))
    deg = degenerate_rays(vh, *N)
    y64[deg] = 0.0
    x = torch.from_numpy(x64).float().cuda()
    y = torch.from_numpy(y64).float().cuda()
    m = torch.from_numpy((rng.random(N + (FEW,)) < 0.2)).to(torch.uint8).cuda() if masked else None
    mh = siddon.pack_map_header(ch)
    few, many = siddon.upload_views(vh), siddon.upload_views(vh * TIMES)
    T = FEW * TIMES
    mm = None if m is None else m.repeat(1, 1, TIMES)

    want = torch.zeros(N + (FEW,), device="cuda")
    siddon.run_device("pj", want, x, few, mh, FEW, m, "sun")
    added = torch.ones_like(want)                        # the product and the sum round once
    siddon.run_device("pj", added, x, few, mh, FEW, m, "sun")
    ref = InfoArray(shape=N + (FEW,), header=[dict(h) for h in vh], dtype=np.float64)
    mask = None if m is None else m.cpu().numpy().astype(np.float64)
    oracle.projector(ref, InfoArray(data=x.cpu().numpy().astype(np.float64), header=dict(ch)), mask=mask, obstacle="sun")
    rel, norm = image_errors(want.cpu().numpy(), ref, exclude=deg)
    assert rel <= IMG_TOL and norm <= IMG_TOL, (rel, norm)
    # views innermost, then views outermost
    for order in ((0, 1, 2), (2, 0, 1)):
        shape = [(N + (T,))[k] for k in order]
        img = torch.full(shape, 7.0, device="cuda").permute([order.index(k) for k in range(3)])
        siddon.run_device("pj", img, x, many, mh, T, mm, "sun", overwrite=True)
        assert torch.equal(img.reshape(N + (TIMES, FEW)), want[:, :, None, :].expand(-1, -1, TIMES, -1))
        img.fill_(1.0)
        siddon.run_device("pj", img, x, many, mh, T, mm, "sun")
        assert torch.equal(img.reshape(N + (TIMES, FEW)), added[:, :, None, :].expand(-1, -1, TIMES, -1))

    cref = InfoArray(shape=n, header=dict(ch), dtype=np.float64)
    oracle.backprojector(InfoArray(data=y.cpu().numpy().astype(np.float64), header=[dict(h) for h in vh]), cref,
                         mask=mask, obstacle="sun")
    # one copy of each view carries data (a sum of all copies would round with
    # its 4e5 terms), at different places of the launch
    spread = torch.zeros(N + (TIMES, FEW), device="cuda")
    for v in range(FEW):
        spread[:, :, (37 * v) % TIMES, v] = y[:, :, v]
    for tab, data, mk, views in ((few, y, m, FEW), (many, spread.reshape(N + (T,)), mm, T)):
        cube = torch.zeros(n, device="cuda")
        siddon.run_device("bpj", data, cube, tab, mh, views, mk, "sun")
        rel, norm = cube_errors(cube.cpu().numpy(), cref, float(y64.max()), ch["CDELT1"])
        assert rel <= CUBE_TOL and norm <= CUBE_TOL, (views, rel, norm)
