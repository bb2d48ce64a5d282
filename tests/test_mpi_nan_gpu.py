"""vlp4d_mpi advections whose feet are not numbers: a NaN or an infinity in the
field, in f (which reaches the field through the moment) or in dt is a foot out
of range like any other.  The points receive 0, vlp4d_check reports it, all
other points keep their bits, and the context goes on working."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import IC_SLD10, MpiRestatement, interior

pytestmark = pytest.mark.gpu

L, VMAX, DT = 4 * np.pi, 9.0, 0.02
SHAPES = [(10, 10, 10, 10), (33, 13, 11, 10)]


def _ctx(pkg, n):
    return pkg.Context(pkg.Domain(list(n), [0.0, 0.0, -VMAX, -VMAX], [L, L, VMAX, VMAX], DT, 2, 10), "f64")


def _range_error(pkg, ctx):
    with pytest.raises(pkg.vlp4d.Vlp4dError) as e:
        ctx.check()
    assert e.value.code == pkg.vlp4d.ERR_RANGE
    ctx.check()  # reported once


@pytest.mark.parametrize("kernels", ["auto", "fused", "generic"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n", SHAPES)
def test_field_not_finite(pkg, cuda, monkeypatch, n, value, kernels):
    torch = cuda
    monkeypatch.setenv("VLP4D_KERNELS", kernels)
    rest = MpiRestatement(n, (0, 0, -VMAX, -VMAX), (L, L, VMAX, VMAX), DT, 10)
    rng = np.random.default_rng(sum(n))
    c4 = 1 + rng.random(rest.init_halo(IC_SLD10).shape)  # no sum of its taps is 0
    ex, ey = (0.4 * rng.uniform(-1, 1, (n[1], n[0])) for _ in range(2))
    want, err = rest.advect_4d(c4, ex, ey)
    assert not err
    with _ctx(pkg, n) as ctx:
        for field, at in ((ctx.ex, (4, 7)), (ctx.ey, (n[1] - 1, 0))):
            ctx.ex.copy_(torch.from_numpy(ex).cuda())
            ctx.ey.copy_(torch.from_numpy(ey).cuda())
            field[at] = value
            c = torch.from_numpy(c4).cuda()
            ctx.mpi_advect_4d(c, ctx.mpi_empty(), DT)
            _range_error(pkg, ctx)
            got, ref = interior(c.cpu().numpy()), interior(want)
            assert ((got == ref) | (got == 0.0)).all()
            # The three by three predictor points around the value, no more.
            lost = (got == 0.0).any(axis=(0, 1))
            assert lost[at] and lost.sum() <= 25


@pytest.mark.parametrize("dt", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n", SHAPES)
def test_dt_not_finite(pkg, cuda, n, dt):
    torch = cuda
    with _ctx(pkg, n) as ctx:
        ctx.ex.fill_(0.1)
        ctx.ey.fill_(-0.1)
        for name in ("mpi_advect_4d", "mpi_advect_2d"):
            c = torch.ones(tuple(ctx.mpi_empty().shape), dtype=torch.float64, device="cuda")
            getattr(ctx, name)(c, ctx.mpi_empty(), dt)
            _range_error(pkg, ctx)


@pytest.mark.parametrize("value", [np.nan, np.inf, 1e308])
def test_fused_step_of_f_not_finite(pkg, cuda, value):
    torch = cuda
    n = SHAPES[1]
    rest = MpiRestatement(n, (0, 0, -VMAX, -VMAX), (L, L, VMAX, VMAX), DT, 10)
    f0 = rest.init_halo(IC_SLD10)
    with _ctx(pkg, n) as ctx:
        bad = torch.from_numpy(f0).cuda()
        bad[5, 6, 7, 8] = value
        ctx.mpi_step(bad, ctx.mpi_empty(), 1)
        _range_error(pkg, ctx)
        # The next run on good data is right.
        out = ctx.mpi_run(torch.from_numpy(f0).cuda(), ctx.mpi_empty(), 1)
        ctx.check()
        got, want = interior(out.cpu().numpy()), interior(rest.run_mpi(f0, 1)[0])
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
