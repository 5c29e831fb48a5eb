"""Workspace of the segmented inner product (csrc/packed.cu): its parts go
through the caller's workspace, never through another CTA's shared memory,
which may only be written once that CTA is known to run."""
import ctypes
import os
import re

import pytest

from tomograpy_gb300 import _build, _lib


@pytest.fixture(scope="module")
def lib(built):
    from tomograpy_gb300.batch import _bind
    return _bind(_lib.load())


def test_workspace_holds_every_part(lib):
    """32 partials of 8 parts per segment up to 15 segments, 32 partials from
    there (a CTA then sums the parts itself)."""
    size = lib.tg_segmented_workspace_bytes
    assert [size(n) for n in (0, 1, 3, 15)] == [0, 2048, 3 * 2048, 15 * 2048]
    assert [size(n) for n in (16, 17, 65535)] == [16 * 256, 17 * 256, 65535 * 256]


def test_no_remote_shared_memory_without_a_barrier_before():
    """A store to another CTA's shared memory needs a cluster barrier before it
    as well as one behind it."""
    for name in sorted(os.listdir(_build.CSRC)):
        with open(os.path.join(_build.CSRC, name)) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        for kernel in re.split(r"__global__", code)[1:]:
            remote = re.search(r"map_shared_rank|mapa\.|shared::cluster", kernel)
            if remote:
                assert re.search(r"\.sync\(\)|barrier_wait|barrier\.cluster\.wait", kernel[:remote.start()]), name


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 15, 16])
def test_small_workspace_gives_the_same_bits(lib, n):
    """256 bytes per segment were enough at all times: they still are, with the
    same sums, and nothing is written behind the size that was passed."""
    import torch
    lengths = [0, 1, 1023, 1024, 1025, 32768 * 8, 32768 * 8 + 1, 70001][:max(1, n)]
    bounds, at = [], 1
    for k in range(n):
        bounds += [at, at + lengths[(k + 1) % len(lengths)]]
        at = bounds[-1] + 3
    g = torch.Generator(device="cuda").manual_seed(n)
    a, b = (torch.randn(at, generator=g, device="cuda") for _ in range(2))
    seg = torch.tensor(bounds, dtype=torch.int64, device="cuda")
    out = []
    for size in (lib.tg_segmented_workspace_bytes(n), 256 * n):
        ws = torch.full((size // 8 + 64,), 7.0, dtype=torch.float64, device="cuda")
        got = torch.full((n,), 3.0, dtype=torch.float64, device="cuda")
        args = [ctypes.c_void_p(t.data_ptr()) for t in (a, b, seg)]
        rest = [n, ctypes.c_void_p(got.data_ptr()), ctypes.c_void_p(ws.data_ptr())]
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(lib.tg_segmented_dot_f32(*args, *rest, size, st))
        assert bool((ws[size // 8:] == 7.0).all())
        out.append(got)
    assert torch.equal(out[0], out[1])
    for k in range(n):
        x, y = (t[bounds[2 * k]:bounds[2 * k + 1]].double() for t in (a, b))
        # sums of fewer than 2^12 additions, each within 2^-53 of its size
        assert abs(float(out[0][k] - (x * y).sum())) <= 2.0 ** -40 * float((x * y).abs().sum())
    with pytest.raises(Exception):
        _lib.check(lib.tg_segmented_dot_f32(*args, *rest, 256 * n - 8, st))
