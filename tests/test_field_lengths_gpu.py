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


@pytest.mark.parametrize("idcase", [10, 110])
@pytest.mark.parametrize("nxy", [(9, 16), (12, 12), (24, 24), (31, 29), (25, 27), (45, 39), (60, 60), (36, 48), (48, 44), (72, 60)])
def test_solve_error(pkg, cuda, nxy, idcase):
    """Ex against the solve in extended precision, for densities whose mean is
    taken out (idcase 10) and left in (110): 4 units in the last place of the
    largest value, rms (a transform rounds each of its some ten steps by 0.3
    units), whatever the mean beside the perturbation."""
    import scipy.fft

    torch = cuda
    nx, ny = nxy
    ld, L = np.longdouble, 12.5
    f = lambda n: np.where(np.arange(n) <= n // 2, np.arange(n), np.arange(n) - n).astype(ld)  # noqa: E731
    kx, ky = np.meshgrid(2 * ld(np.pi) / ld(L) * np.where(2 * f(nx) == nx, 0, f(nx)), 2 * ld(np.pi) / ld(L) * f(ny))
    k2 = np.meshgrid(f(nx), f(ny))
    k2 = (2 * ld(np.pi) / ld(L)) ** 2 * (k2[0] ** 2 + k2[1] ** 2)
    k2[0, 0] = 1
    dom = pkg.Domain([nx, ny, 8, 8], [0.0, 0.0, -6.0, -6.0], [L, L, 6.0, 6.0], 0.1, 1, idcase)
    err = []
    with pkg.Context(dom, "f64") as ctx:
        for seed in range(4):
            rho = 1 + 0.1 * np.random.default_rng(seed).standard_normal((ny, nx))
            r = scipy.fft.fft2((rho.astype(ld) - (idcase == 10)).astype(np.clongdouble)) / k2
            r[0, 0] = 0
            want = scipy.fft.ifft2(-1j * kx * r).real
            ctx.rho.copy_(torch.from_numpy(rho).cuda())
            ctx.field_poisson()
            ctx.check()
            got = ctx.ex.cpu().numpy().astype(ld)
            err.append(float(np.sqrt(np.mean((got - want) ** 2)) / np.abs(want).max()))
    assert np.mean(err) <= 4 * 1.11e-16, err
