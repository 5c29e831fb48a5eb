"""Segmented vector kernels of CG (csrc/packed.cu) at lengths around their
16-byte accesses and shares, at starts that are not 16-byte aligned, and with
few segments (a cluster per partial) and many (a CTA per partial): the updates
against single float32 operations, the inner product against float64 within
the rounding of its float64 sums, and bitwise equal wherever the segment
stands."""
import numpy as np
import pytest

from tomograpy_gb300 import cg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

LENGTHS = [0, 1, 3, 4, 5, 1023, 1024, 8193, 32768 * 8 - 1, 32768 * 8 + 3, 600001]


@pytest.fixture(scope="module", autouse=True)
def _build(built):
    return built


@pytest.mark.parametrize("copies", [1, 20])
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_segments(copies, shift):
    lengths = LENGTHS if copies == 1 else LENGTHS[:9] * 3
    bounds, at = [], shift
    for n in lengths:
        bounds += [at, at + n]
        at += n + 2
    g = torch.Generator(device="cuda").manual_seed(7)
    v = [torch.randn(at, generator=g, device="cuda") for _ in range(4)]
    n = len(lengths)
    ops = cg.SegmentOps(bounds, "cuda")
    out = ops.dot(v[0], v[1], torch.zeros(n, dtype=torch.float64, device="cuda"))
    for k in range(n):
        a, b = (t[bounds[2 * k]:bounds[2 * k + 1]].clone() for t in v[:2])
        ref = float((a.double() * b.double()).sum())
        scale = float((a.double() * b.double()).abs().sum())
        # fewer than 2^12 additions deep in either order
        assert abs(float(out[k]) - ref) <= 2.0 ** -40 * scale
        if lengths[k]:
            alone = cg.SegmentOps([0, lengths[k]], "cuda").dot(a, b, torch.zeros(1, dtype=torch.float64, device="cuda"))
            assert float(alone[0]) == float(out[k])
    num = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) + 0.5
    den = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) + 0.5
    f = (num / den).float().cpu().numpy().astype(np.float64)
    old = [t.cpu().numpy().astype(np.float64) for t in v]
    inside = np.zeros(at, bool)
    fac = np.zeros(at)
    for k in range(n):
        inside[bounds[2 * k]:bounds[2 * k + 1]] = True
        fac[bounds[2 * k]:bounds[2 * k + 1]] = f[k]
    x, r, p = (v[k].clone() for k in (0, 1, 2))
    ops.update_x(x, r, p, v[3], num, den)
    # one float32 multiply-add each: the exact value rounded once (float64 holds
    # the product exactly, its sum to 2^-53)
    for got, want in ((x, old[0] + fac * old[2]), (r, old[1] - fac * old[3])):
        got = got.cpu().numpy().astype(np.float64)
        assert np.all(np.abs(got - want)[inside] <= 2.0 ** -23 * np.abs(want)[inside] + 1e-14)
    assert np.array_equal(x.cpu().numpy()[~inside], v[0].cpu().numpy()[~inside])
    p2, rr = v[2].clone(), den.clone()
    ops.update_p(p2, v[1], rr, num)
    want = old[1] + fac * old[2]
    assert np.all(np.abs(p2.cpu().numpy() - want)[inside] <= 2.0 ** -23 * np.abs(want)[inside] + 1e-14)
    assert torch.equal(rr, num)
    y = v[0].clone()
    ops.axpby(y, v[1], 0.25, 1.0)
    want = old[0] + 0.25 * old[1]
    assert np.all(np.abs(y.cpu().numpy() - want)[inside] <= 2.0 ** -23 * np.abs(want)[inside] + 1e-14)
    assert np.array_equal(y.cpu().numpy()[~inside], v[0].cpu().numpy()[~inside])
    ops.axpby(y, None, 1.0, 0.0)
    assert not y.cpu().numpy()[inside].any()
