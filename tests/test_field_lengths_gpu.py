"""The cluster field solve at lengths with two factors, primes, odd rows and
row counts that leave CTAs short or empty, against the cuFFT path of the same
entry point (1e-13 of the field's maximum, as for the other lengths); the
moment in one launch against the FP64 sum of the planes."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxy", [(2, 2), (3, 5), (9, 7), (17, 16), (45, 39), (43, 41), (72, 60), (49, 15), (31, 100), (128, 9)])
def test_solve_matches_cufft(pkg, cuda, monkeypatch, nxy):
    torch = cuda
    nx, ny = nxy
    dom = pkg.landau_domain((nx, ny, 8, 8), dt=0.1, nbiter=1)
    gen = torch.Generator().manual_seed(nx * 1000 + ny)
    rho = (1.0 + 0.1 * torch.rand((ny, nx), generator=gen, dtype=torch.float64)).cuda()
    got = {}
    for mode in ("", "cufft"):
        monkeypatch.setenv("VLP4D_FIELD", mode)
        with pkg.Context(dom, "f64") as ctx:
            ctx.rho.copy_(rho)
            ctx.field_poisson()
            ctx.check()
            got[mode] = [t.clone() for t in (ctx.rho, ctx.ex, ctx.ey)]
    # The fields share one scale (a grid of two columns has no Ex of its own).
    scale = max(float(t.abs().max()) for t in got["cufft"])
    for a, b in zip(got[""], got["cufft"]):
        assert float((a - b).abs().max()) <= 1e-13 * scale


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("n", [(1, 1, 1, 1), (5, 3, 2, 3), (16, 16, 16, 16), (33, 7, 31, 33), (90, 91, 4, 4), (91, 91, 4, 4),
                               (4, 4, 32, 33)])
def test_moment(pkg, cuda, n, dtype):
    torch = cuda
    dom = pkg.landau_domain(n)
    with pkg.Context(dom, dtype) as ctx:
        f = torch.rand(ctx.f_shape, generator=torch.Generator().manual_seed(1), dtype=torch.float64).to(ctx.torch_dtype).cuda()
        ctx.field_rho(f)
        want = f.double().sum((0, 1)) * dom.dx[2] * dom.dx[3]
        # At most 2 nv roundings of sums below nv.
        assert float((ctx.rho - want).abs().max()) <= 2 * 1.2e-16 * (n[2] * n[3]) ** 2 * dom.dx[2] * dom.dx[3] + 1e-16


def test_calls_go_to_the_current_stream(pkg, cuda):
    """Without a stream argument a call runs on PyTorch's current stream, the
    default one, a side stream and the default one again."""
    torch = cuda
    ptr = pkg.vlp4d._stream_ptr
    side = torch.cuda.Stream()
    assert ptr(None) == torch.cuda.current_stream().cuda_stream
    with torch.cuda.stream(side):
        assert ptr(None) == side.cuda_stream
    assert ptr(None) == torch.cuda.current_stream().cuda_stream
    assert ptr(side) == side.cuda_stream
