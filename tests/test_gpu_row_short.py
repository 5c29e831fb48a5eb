"""Short rays of a row-walk view (csrc/siddon_rows.cuh): rays that leave the
cube through a face of its axis 2 soon after they entered, and rays that enter
it so just before they leave, with chords of 1.5e-3 to 0.09 of the row's 3 radii.

Tolerance: they are measured from the middle of their own chord: each of a few crossings is rounded at 2^-25 of the chord, each
product, sum and 1 / cos(lambda) at 2^-24, the entry is exact to 1e-11 radii:
below 10 * 2^-24 = 6e-7 of the chord in all, 1e-6 here."""
import numpy as np
import pytest

from tomograpy_gb300 import headers as H
from tomograpy_gb300 import lo_wrapper
from tomograpy_gb300.infoarray import InfoArray

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

N, n = (5, 60), (48, 48, 48)


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def _geometry(below):
    ch = H.centered_cubic_map_header([3.0, 3.0, 3.0], n, dtype=np.float32)
    if not below:                                  # a cube that begins at z = 1.5
        ch["CRPIX3"] = -24.0
        H.map_borders(ch)
    # columns whose ray passes z = 1.5 a distance c behind its entry at x = 1.5
    # (below), or before its exit at x = -1.5
    c = np.array([1.5e-3, 0.09])
    lam = np.arctan(1.5 / (213.5 + c if below else 216.5 - c))
    h = H.centered_image_header(1e-3, N, dtype=np.float32)
    h.update({"CDELT1": 1e-4, "CRVAL1": 4e-5, "CRPIX2": 1.0, "CRVAL2": lam[0], "CDELT2": (lam[1] - lam[0]) / (N[1] - 1),
              "LON": 0.0, "LAT": 0.0, "ROL": 0.0, "D": 215.0, "M1": 215.0, "M2": 0.0, "M3": 0.0})
    H.header_rotation_matrix(h)
    return ch, [h]


@pytest.mark.parametrize("below", [True, False])
def test_short_rays(below):
    import oracle
    ch, vh = _geometry(below)
    x = (0.2 + np.random.default_rng(4).random(n)).astype(np.float32)

    def project(v):
        out = InfoArray(shape=N + (1,), header=[dict(h) for h in vh], dtype=np.float64)
        oracle.projector(out, InfoArray(data=v.astype(np.float64), header=dict(ch)))
        return np.asarray(out)

    ref, chord = project(x), project(np.ones(n))
    assert chord.min() > 1e-3 and 0.08 < chord.max() < 0.0935
    op = lo_wrapper.siddon_lo(vh, ch, dtype=np.float32)
    got = op.project(torch.from_numpy(x)).cpu().numpy().astype(np.float64)
    err = (np.abs(got - ref) / ref).max()
    assert err <= 1e-6, err
    for det in (False, True):
        op = lo_wrapper.siddon_lo(vh, ch, dtype=np.float32, deterministic=det)
        for i, j in ((0, 0), (1, 1), (2, 7), (4, 30), (3, 59)):
            y = np.zeros(N + (1,), np.float32)
            y[i, j] = 1.0
            cref = InfoArray(shape=n, header=dict(ch), dtype=np.float64)
            oracle.backprojector(InfoArray(data=y.astype(np.float64), header=[dict(h) for h in vh]), cref)
            got = op.backproject(torch.from_numpy(y)).cpu().numpy()
            assert np.abs(got - np.asarray(cref)).max() <= 1e-6 * chord[i, j, 0], (det, i, j)
