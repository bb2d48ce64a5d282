"""The tiled vlp4d_mpi 4D advection at the edges of its tiles: x tiles of 32
and their remainders, groups of four y with one to four cells, partial vx
tiles and vy segments, and feet on either side of every grid point.

The reference-order entry point is compared bit for bit with the restated
reference, under fields that leave all first taps within one cell (the tiled
sums), that change sign from point to point (every mixture of first taps) and
that push feet several cells away (the cell-by-cell route).  The fused step is
held to the tolerance of the other fused-step tests (1e-12 of max|f|).
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import IC_SLD10, MpiRestatement, interior

pytestmark = pytest.mark.gpu

L, VMAX, DT = 4 * np.pi, 9.0, 0.02
SHAPES = [(10, 10, 10, 10), (33, 13, 11, 10), (32, 12, 16, 11), (35, 10, 10, 21), (64, 11, 13, 10), (12, 34, 10, 12)]


def _dom(pkg, n, nbiter=2):
    return pkg.Domain(list(n), [0.0, 0.0, -VMAX, -VMAX], [L, L, VMAX, VMAX], DT, nbiter, 10)


@pytest.mark.parametrize("cells", [0.0, 0.4, 2.7])
@pytest.mark.parametrize("n", SHAPES)
def test_advect_4d_bit_identical(pkg, cuda, n, cells):
    torch = cuda
    rest = MpiRestatement(n, (0, 0, -VMAX, -VMAX), (L, L, VMAX, VMAX), DT, 10)
    rng = np.random.default_rng(sum(n))
    # The stage takes any coefficients: random ones show every tap.
    c4 = rng.standard_normal(rest.init_halo(IC_SLD10).shape)
    # Displacements of up to `cells` cells in vx and vy.
    scale = cells * (2 * VMAX / max(n[2], n[3])) / DT
    ex, ey = (scale * rng.uniform(-1, 1, (n[1], n[0])) for _ in range(2))
    want, err = rest.advect_4d(c4, ex, ey)
    with pkg.Context(_dom(pkg, n), "f64") as ctx:
        ctx.ex.copy_(torch.from_numpy(ex).cuda())
        ctx.ey.copy_(torch.from_numpy(ey).cuda())
        c = torch.from_numpy(c4).cuda()
        tmp = ctx.mpi_empty()
        ctx.mpi_advect_4d(c, tmp, DT)
        if err:  # the strongest field pushes some x feet of the 64-column grid out of range
            with pytest.raises(pkg.vlp4d.Vlp4dError) as e:
                ctx.check()
            assert e.value.code == pkg.vlp4d.ERR_RANGE
        else:
            ctx.check()
        assert np.array_equal(c.cpu().numpy(), want)
        assert np.array_equal(tmp.cpu().numpy(), c4)


@pytest.mark.parametrize("n", SHAPES)
def test_fused_step(pkg, cuda, n):
    torch = cuda
    rest = MpiRestatement(n, (0, 0, -VMAX, -VMAX), (L, L, VMAX, VMAX), DT, 10)
    f0 = rest.init_halo(IC_SLD10)
    fr, diags, _, _ = rest.run_mpi(f0, 2)
    with pkg.Context(_dom(pkg, n), "f64") as ctx:
        out = ctx.mpi_run(torch.from_numpy(f0).cuda(), ctx.mpi_empty(), 2)
        ctx.check()
        nrj, _ = ctx.diags_read()
        _, _, l2 = ctx.diags_read_ext()
        got, want = interior(out.cpu().numpy()), interior(fr)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
    np.testing.assert_allclose(nrj, diags[:, 0], rtol=0, atol=1e-11)
    np.testing.assert_allclose(l2, diags[:, 4], rtol=1e-12)


@pytest.mark.parametrize("n", [(10, 10, 10, 10), (33, 10, 11, 12), (10, 27, 10, 13), (12, 11, 30, 10)])
def test_halo_fill_bit_identical(pkg, cuda, n):
    torch = cuda
    rest = MpiRestatement(n, (0, 0, -VMAX, -VMAX), (L, L, VMAX, VMAX), DT, 10)
    f0 = np.random.default_rng(sum(n)).standard_normal(rest.init_halo(IC_SLD10).shape)
    with pkg.Context(_dom(pkg, n), "f64") as ctx:
        f = torch.from_numpy(f0).cuda()
        ctx.mpi_halo_fill(f)
        assert np.array_equal(f.cpu().numpy(), rest.halo_fill(f0))


LONG = [(72, 10, 10, 10), (10, 102, 10, 10), (140, 11, 10, 10), (10, 280, 10, 10), (10, 10, 75, 10), (10, 10, 10, 120),
        (11, 10, 150, 10), (10, 10, 10, 300)]
# Beyond the lines the restated reference holds (512 points).
LONGEST = [(10, 560, 10, 10), (10, 10, 560, 10)]


@pytest.mark.parametrize("n", LONG + LONGEST)
def test_fused_step_long_lines(pkg, cuda, n):
    """Every split of the prefilter's lines into segments, in each dimension
    (the boxes grow with the grid so that no shift exceeds a cell); the longest
    against the reference-order entry points."""
    torch = cuda
    Lx, Ly = (L * max(1.0, n[d] / 60) for d in (0, 1))
    rest = MpiRestatement(n, (0, 0, -VMAX, -VMAX), (Lx, Ly, VMAX, VMAX), DT, 10)
    f0 = rest.init_halo(IC_SLD10)
    dom = pkg.Domain(list(n), [0.0, 0.0, -VMAX, -VMAX], [Lx, Ly, VMAX, VMAX], DT, 2, 10)
    with pkg.Context(dom, "f64") as ctx:
        out = ctx.mpi_run(torch.from_numpy(f0).cuda(), ctx.mpi_empty(), 1)
        ctx.check()
        got = interior(out.cpu().numpy())
        if n in LONGEST:
            half, tmp = torch.from_numpy(f0).cuda(), ctx.mpi_empty()
            ctx.mpi_halo_fill(half)
            ctx.mpi_spline_xy(half)
            new = half.clone()
            ctx.mpi_advect_2d(half, tmp, 0.5 * DT)
            ctx.mpi_field(half)
            ctx.mpi_spline_vxvy(new)
            ctx.mpi_advect_4d(new, tmp, DT)
            ctx.check()
            want = interior(new.cpu().numpy())
        else:
            want = interior(rest.run_mpi(f0, 1)[0])
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


def _split_edges():
    """Line lengths n around every split of n + 4 points into G segments of S:
    one point short of it, exact, one beyond, and exact without the first
    segment (the second one then starts at the line's first point)."""
    out = set()
    for S, G in ((5, 8), (9, 8), (13, 8), (17, 8), (17, 16), (17, 32)):
        out |= {S * G - 5, S * G - 4, S * G - 3, S * (G - 1) - 4}
    return sorted(out)


# (The fused step takes up to 512 points along x.)
@pytest.mark.parametrize("dim,n", [(d, n) for d in range(4) for n in _split_edges() if d or n <= 512])
def test_fused_step_split_edges(pkg, cuda, dim, n):
    """The prefilter's lines at the edges of their splits into segments, along
    each dimension, against the restated reference (the reference-order entry
    points beyond its 512 points)."""
    torch = cuda
    size = [10, 11, 10, 12]
    size[dim] = n
    Lx, Ly = (L * max(1.0, size[d] / 60) for d in (0, 1))
    rest = MpiRestatement(tuple(size), (0, 0, -VMAX, -VMAX), (Lx, Ly, VMAX, VMAX), DT, 10)
    f0 = rest.init_halo(IC_SLD10)
    # No symmetry about the box's ends: the boundary sums of both differ.
    x, y = (np.arange(size[d] + 6) - 3 for d in (0, 1))
    f0 *= (1 + 0.3 * np.sin(2 * np.pi * x / size[0] + 0.7))[None, None, None, :]
    f0 *= (1 + 0.2 * np.sin(2 * np.pi * y / size[1] - 0.4))[None, None, :, None]
    dom = pkg.Domain(size, [0.0, 0.0, -VMAX, -VMAX], [Lx, Ly, VMAX, VMAX], DT, 2, 10)
    with pkg.Context(dom, "f64") as ctx:
        out = ctx.mpi_run(torch.from_numpy(f0).cuda(), ctx.mpi_empty(), 1)
        ctx.check()
        got = interior(out.cpu().numpy())
        if n + 6 > 512:
            half, tmp = torch.from_numpy(f0).cuda(), ctx.mpi_empty()
            ctx.mpi_halo_fill(half)
            ctx.mpi_spline_xy(half)
            new = half.clone()
            ctx.mpi_advect_2d(half, tmp, 0.5 * DT)
            ctx.mpi_field(half)
            ctx.mpi_spline_vxvy(new)
            ctx.mpi_advect_4d(new, tmp, DT)
            ctx.check()
            want = interior(new.cpu().numpy())
        else:
            want = interior(rest.run_mpi(f0, 1)[0])
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("n", [(10, 10, 10, 10), (10, 26, 10, 11), (32, 8 + 3, 10, 10), (33, 17, 11, 10), (65, 12, 10, 10),
                               (16, 257, 10, 10), (11, 300, 10, 10)])
def test_advect_2d_bit_identical(pkg, cuda, n):
    """The 2D advection at the edges of its (x, y) tiles."""
    torch = cuda
    Lx, Ly = (L * max(1.0, n[d] / 60) for d in (0, 1))
    rest = MpiRestatement(n, (0, 0, -VMAX, -VMAX), (Lx, Ly, VMAX, VMAX), DT, 10)
    c4 = np.random.default_rng(sum(n)).standard_normal(rest.init_halo(IC_SLD10).shape)
    want, err = rest.advect_2d(c4, 0.5 * DT)
    assert not err
    dom = pkg.Domain(list(n), [0.0, 0.0, -VMAX, -VMAX], [Lx, Ly, VMAX, VMAX], DT, 2, 10)
    with pkg.Context(dom, "f64") as ctx:
        c, tmp = torch.from_numpy(c4).cuda(), ctx.mpi_empty()
        ctx.mpi_advect_2d(c, tmp, 0.5 * DT)
        ctx.check()
        assert np.array_equal(c.cpu().numpy(), want)


@pytest.mark.parametrize("kernels", ["fused", "generic"])
@pytest.mark.parametrize("cells", [0.4, 2.7])
@pytest.mark.parametrize("n", SHAPES + [(28, 11, 10, 10), (26, 19, 10, 12), (45, 10, 12, 10)])
def test_advect_4d_both_routes(pkg, cuda, monkeypatch, n, cells, kernels):
    """The reference-order 4D advection by tiles and by one thread per cell,
    whichever the size would choose."""
    monkeypatch.setenv("VLP4D_KERNELS", kernels)
    test_advect_4d_bit_identical(pkg, cuda, n, cells)
