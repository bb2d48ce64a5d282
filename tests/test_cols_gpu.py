"""The sweeps by columns (any shape and alignment) against one thread per
output: the same arithmetic per output, so the same bits, in every direction,
type and pair, at tile and strip edges, extents below the stencil's width,
offsets of several periods and unaligned buffers."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2, 3, 8), (5, 7, 3, 2), (13, 17, 9, 7), (33, 16, 5, 11), (45, 39, 11, 5), (127, 33, 3, 4), (129, 5, 2, 9),
          (257, 18, 4, 3), (6, 100, 7, 6)]


def _ctx(pkg, monkeypatch, n, dtype, mode):
    monkeypatch.setenv("VLP4D_KERNELS", mode)
    dom = pkg.Domain(list(n), [0.0, 0.0, -6.0, -6.0], [4 * np.pi, 4 * np.pi, 6.0, 6.0], 0.1, 4, 10)
    return pkg.Context(dom, dtype)


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("n", SHAPES)
def test_same_bits_as_cell_per_thread(pkg, cuda, monkeypatch, n, dtype):
    torch = cuda
    g = torch.Generator().manual_seed(sum(n))
    with _ctx(pkg, monkeypatch, n, dtype, "auto") as ctx, _ctx(pkg, monkeypatch, n, dtype, "generic") as gen:
        f = torch.rand(ctx.f_size + 1, generator=g, dtype=torch.float64).to(ctx.torch_dtype).cuda()
        # Fields of up to a few cells' shift, signs mixed.
        for which in (ctx, gen):
            h = torch.Generator().manual_seed(7)
            which.ex.copy_((torch.rand(n[1], n[0], generator=h, dtype=torch.float64) - 0.5) * 8)
            which.ey.copy_((torch.rand(n[1], n[0], generator=h, dtype=torch.float64) - 0.5) * 8)
        for shift in (0, 1):  # the second buffer starts off the 16-byte boundary
            src = f[shift:shift + ctx.f_size].view(ctx.f_shape)
            for name in ("advect_x", "advect_y", "advect_vx", "advect_vy", "advect_xy", "advect_xy_moment", "advect_vxvy"):
                for dt in (0.3, -2.9):
                    out, want = (torch.full_like(f, 9.0)[shift:shift + ctx.f_size].view(ctx.f_shape) for _ in range(2))
                    getattr(ctx, name)(src, out, dt)
                    getattr(gen, name)(src, want, dt)
                    ctx.check()
                    if shift or n[0] % 4 or name[7:9] == "vx" or name == "advect_vy":
                        assert torch.equal(out, want), (name, dt, shift)
                    else:
                        tol = 1e-13 if dtype == "f64" else 2e-6
                        assert float((out - want).abs().max()) <= tol, (name, dt)
                    if name == "advect_xy_moment":
                        # Sums of at most nvx nvy values near 1 in another order.
                        tol = 4e-16 * (n[2] * n[3]) ** 2 if dtype == "f64" else 2e-6 * n[2] * n[3]
                        scale = 12.0 * 12.0 / (n[2] * n[3])
                        assert float((ctx.rho - gen.rho).abs().max()) <= tol * scale


@pytest.mark.parametrize("n", [(13, 17, 9, 7), (45, 39, 11, 5)])
def test_time_loop_matches_separate_steps(pkg, cuda, monkeypatch, n):
    """FP32 loops of such grids: `steps` against single steps, to the rounding
    of the joined half steps (2e-6 of max|f| per joined pass)."""
    torch = cuda
    with _ctx(pkg, monkeypatch, n, "f32", "auto") as ctx:
        f = ctx.empty_f()
        ctx.init_case(f)
        a, b = f.clone(), ctx.empty_f()
        ctx.steps(a, b, 1, 3)
        p, q = f.clone(), ctx.empty_f()
        for it in range(1, 4):
            ctx.step(p, q, it)
            p, q = q, p
        ctx.check()
        assert float((b - p).abs().max()) <= 3 * 2e-6 * float(f.max())


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("n", [(64, 8, 16, 43), (32, 32, 8, 131), (16, 16, 32, 7), (64, 64, 64, 61)])
def test_uneven_vy_segments(pkg, cuda, monkeypatch, n, dtype):
    """The v-slab pass where its vy segments do not divide nvy (the last one is
    shorter), forced, against one thread per output; tolerances as for the
    other fused-against-generic comparisons."""
    torch = cuda
    tol = 1e-14 if dtype == "f64" else 2e-7
    with _ctx(pkg, monkeypatch, n, dtype, "fused") as fz, _ctx(pkg, monkeypatch, n, dtype, "generic") as gen:
        f = fz.empty_f()
        fz.init_case(f)
        for which in (fz, gen):
            h = torch.Generator().manual_seed(3)
            which.ex.copy_(torch.randn(n[1], n[0], generator=h, dtype=torch.float64) * 3)
            which.ey.copy_(torch.randn(n[1], n[0], generator=h, dtype=torch.float64) * 3)
        for name in ("advect_vx", "advect_vy", "advect_vxvy"):
            out, want = fz.empty_f(), gen.empty_f()
            getattr(fz, name)(f, out, 0.2)
            getattr(gen, name)(f, want, 0.2)
            fz.check()
            assert float((out - want).abs().max()) <= tol * float(want.abs().max()), name


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("n", [(64, 37, 8, 9), (32, 74, 8, 8), (72, 55, 8, 8), (128, 127, 8, 8), (20, 21, 8, 8), (256, 13, 8, 8)])
def test_overlapping_row_chunks(pkg, cuda, monkeypatch, n, dtype):
    """The plane passes where the chunk height does not divide ny (the last
    chunk overlaps the one before), forced, against one thread per output, and
    the joined pass against two passes; tolerances as for the other shapes."""
    torch = cuda
    tol = 1e-14 if dtype == "f64" else 2e-7
    with _ctx(pkg, monkeypatch, n, dtype, "fused") as fz, _ctx(pkg, monkeypatch, n, dtype, "generic") as gen:
        f = fz.empty_f()
        fz.init_case(f)
        for name in ("advect_x", "advect_y", "advect_xy", "advect_xy_moment"):
            out, want = (torch.full_like(f, 9.0) for _ in range(2))
            getattr(fz, name)(f, out, 0.21)
            getattr(gen, name)(f, want, 0.21)
            fz.check()
            assert float((out - want).abs().max()) <= tol * float(want.abs().max()), name
        assert float((fz.rho - gen.rho).abs().max()) <= (1e-13 if dtype == "f64" else 1e-6) * float(gen.rho.abs().max())
        out, half, want = (torch.full_like(f, 9.0) for _ in range(3))
        fz.advect_xyxy(f, out, 0.21)
        fz.advect_xy(f, half, 0.21)
        fz.advect_xy_moment(half, want, 0.21)
        fz.check()
        assert float((out - want).abs().max()) <= (1e-13 if dtype == "f64" else 2e-6) * float(want.abs().max())


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("n", [(24, 6, 7, 5), (24, 5, 7, 5), (23, 6, 5, 7), (20, 13, 5, 7), (20, 12, 9, 4), (19, 14, 3, 8), (8, 12, 9, 7),
                               (8, 11, 7, 9), (7, 14, 6, 8), (26, 4, 6, 5), (34, 3, 6, 5), (4, 16, 9, 7), (5, 13, 9, 7), (5, 12, 9, 7),
                               (3, 22, 6, 9), (19, 5, 9, 8), (16, 6, 9, 8), (127, 1, 9, 8), (128, 1, 8, 9), (1, 129, 9, 8)])
def test_routes_on_either_side(pkg, cuda, monkeypatch, n, dtype):
    """Planes just inside and just outside of what the column kernels take."""
    test_same_bits_as_cell_per_thread(pkg, cuda, monkeypatch, n, dtype)
