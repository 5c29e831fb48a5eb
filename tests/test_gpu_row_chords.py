"""Short chords of a row-walk view (csrc/siddon_rows.cuh): whole rows that clip
an edge of the cube (they leave through a face of axis 1 soon after they entered,
or enter through it just before they leave), and rays that do so at a face of
axis 2, in fine cubes and in cubes of voxels much longer than the chord.

Tolerance: entry and exit are exact to 1e-11 radii in double-float, crossings in
between rounded at 2^-25 of the chord each, and product, sum and 1 / cos(lambda)
at 2^-24: below 10 * 2^-24 = 6e-7 of the chord in all, 1e-6 here."""
import numpy as np
import pytest

from tomograpy_gb300 import headers as H
from tomograpy_gb300 import lo_wrapper
from tomograpy_gb300.infoarray import InfoArray

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


def geometry(axis, enters, chords, n):
    """60 rays (rows of the image for axis 1, columns for axis 2) that pass the
    plane 1.5 of that axis a distance c behind x = 1.5 or before x = -1.5."""
    N = (60, 5) if axis == 1 else (5, 60)
    ch = H.centered_cubic_map_header([3.0, 3.0, 3.0], n, dtype=np.float32)
    if enters:                                     # a cube that begins at 1.5
        ch["CRPIX%d" % (axis + 1)] = -n[axis] / 2.0
        H.map_borders(ch)
    c = np.array(chords)
    a = np.arctan(1.5 / (216.5 - c if enters else 213.5 + c))
    long, wide = (1, 2) if axis == 1 else (2, 1)
    h = H.centered_image_header(1e-3, N, dtype=np.float32)
    h.update({"CRPIX%d" % long: 1.0, "CRVAL%d" % long: a[0], "CDELT%d" % long: (a[1] - a[0]) / 59,
              "CDELT%d" % wide: 1e-4, "CRVAL%d" % wide: 4e-5, "LON": 0.0, "LAT": 0.0, "ROL": 0.0, "D": 215.0,
              "M1": 215.0, "M2": 0.0, "M3": 0.0})
    H.header_rotation_matrix(h)
    return ch, [h], N


@pytest.mark.parametrize("n", [(48, 48, 48), (2, 3, 2), (48, 2, 48)])
@pytest.mark.parametrize("enters", [False, True])
@pytest.mark.parametrize("axis, chords", [(1, (1.5e-3, 0.09)), (1, (0.09, 0.37)), (2, (1.5e-3, 0.09)), (2, (0.09, 0.37))])
def test_short_chords(axis, enters, chords, n):
    import oracle
    ch, vh, N = geometry(axis, enters, chords, n)
    x = (0.2 + np.random.default_rng(4).random(n)).astype(np.float32)

    def project(v):
        out = InfoArray(shape=N + (1,), header=[dict(h) for h in vh], dtype=np.float64)
        oracle.projector(out, InfoArray(data=v.astype(np.float64), header=dict(ch)))
        return np.asarray(out)

    ref, chord = project(x), project(np.ones(n))
    assert abs(chord.min() / chords[0] - 1) < 0.05 and abs(chord.max() / chords[1] - 1) < 0.05
    op = lo_wrapper.siddon_lo(vh, ch, dtype=np.float32)
    got = op.project(torch.from_numpy(x)).cpu().numpy().astype(np.float64)
    err = (np.abs(got - ref) / chord).max()
    assert err <= 1e-6, err
    for det in (False, True):
        op = lo_wrapper.siddon_lo(vh, ch, dtype=np.float32, deterministic=det)
        for k in (0, 1, 17, 40, 59):
            i, j = (k, 2) if axis == 1 else (2, k)
            y = np.zeros(N + (1,), np.float32)
            y[i, j] = 1.0
            cref = InfoArray(shape=n, header=dict(ch), dtype=np.float64)
            oracle.backprojector(InfoArray(data=y.astype(np.float64), header=[dict(h) for h in vh]), cref)
            got = op.backproject(torch.from_numpy(y)).cpu().numpy()
            assert np.abs(got - np.asarray(cref)).max() <= 1e-6 * chord[i, j, 0], (det, i, j)
