"""Calls straight after the caller's own event waits: the stream's last work
is a kernel of this library, another stream writes the call's input late, and
the call waits for it by an event only.  Run eagerly, and as a captured graph
whose replays see new inputs.  Same bits as the call on finished inputs."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (32, 32, 16, 24)
CALLS = ["advect_x", "advect_y", "advect_vx", "advect_vy", "advect_xy", "advect_xy_moment", "advect_vxvy", "advect_xyxy",
         "field_rho", "field_poisson", "diags_compute", "step", "steps"]
SLEEP = 4_000_000  # cycles, some 2 ms


def _case(pkg, torch, n, dtype):
    dom = pkg.Domain(list(n), [0.0, 0.0, -6.0, -6.0], [4 * np.pi, 4 * np.pi, 6.0, 6.0], 0.1, 6, 10)
    ctx = pkg.Context(dom, dtype)
    g = torch.Generator().manual_seed(5)
    rnd = lambda *s: torch.rand(*s, generator=g, dtype=torch.float64)  # noqa: E731
    new = [(rnd(*ctx.f_shape).to(ctx.torch_dtype).cuda(), (rnd(n[1], n[0]) - 0.5).cuda()) for _ in range(3)]
    return ctx, new


def _call(ctx, name, f, out):
    if name in ("step", "steps"):
        state = f.clone()  # both overwrite it
        return ctx.step(state, out, 1) if name == "step" else ctx.steps(state, out, 1, 2)
    if name == "field_rho":
        return ctx.field_rho(f)
    if name == "field_poisson":
        return ctx.field_poisson()
    if name == "diags_compute":
        return ctx.diags_compute(1)
    return getattr(ctx, name)(f, out, 0.2)


def _results(torch, ctx, out, name):
    torch.cuda.synchronize()
    got = [out.clone(), ctx.rho.clone(), ctx.ex.clone(), ctx.ey.clone()]
    if name in ("diags_compute", "step", "steps"):
        got += [torch.from_numpy(x[1:3].copy()) for x in ctx.diags_read(4)]
    return got


def _fields(ctx, late, h):
    """The late writer's part: the fields that the call reads."""
    ctx.rho.copy_(h)
    ctx.ex.copy_(3 * h)
    ctx.ey.copy_(2 * h.abs())


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("name", CALLS)
@pytest.mark.parametrize("n", [N, (13, 17, 9, 24)])
@pytest.mark.parametrize("captured", [False, True])
def test_call_after_event(pkg, cuda, n, dtype, name, captured):
    torch = cuda
    ctx, new = _case(pkg, torch, n, dtype)
    main, other = torch.cuda.Stream(), torch.cuda.Stream()
    f, out, prev = (torch.zeros_like(new[0][0]) for _ in range(3))
    src, srch = (t.clone() for t in new[0])
    with ctx:
        if name == "advect_xyxy":
            try:
                ctx.advect_xyxy(f, out, 0.2)
            except pkg.vlp4d.Vlp4dError:
                return  # no joined pass for this shape: refused on the host

        def once():
            # On `main`: a kernel of the library, then the wait for `other`.
            ctx.advect_vxvy(prev, out, 0.2)
            fork, join = torch.cuda.Event(), torch.cuda.Event()
            fork.record(main)
            with torch.cuda.stream(other):
                other.wait_event(fork)
                torch.cuda._sleep(SLEEP)
                f.copy_(src)
                _fields(ctx, True, srch)
                join.record(other)
            main.wait_event(join)
            _call(ctx, name, f, out)

        def fresh(k):
            src.copy_(new[k][0])
            srch.copy_(new[k][1])
            f.zero_()
            out.zero_()
            _fields(ctx, False, torch.zeros_like(srch))
            torch.cuda.synchronize()

        with torch.cuda.stream(main):
            # Finished inputs first: what the late ones have to give, and
            # every table and plan is there before the capture.
            want = []
            for k in range(3):
                fresh(k)
                ctx.advect_vxvy(prev, out, 0.2)
                f.copy_(src)
                _fields(ctx, False, srch)
                torch.cuda.synchronize()
                _call(ctx, name, f, out)
                want.append(_results(torch, ctx, out, name))
            graph = None
            if captured:
                graph = torch.cuda.CUDAGraph()
                torch.cuda.synchronize()
                with torch.cuda.graph(graph, stream=main):
                    once()
            for k in (1, 2, 0):
                fresh(k)
                graph.replay() if captured else once()
                for a, b in zip(_results(torch, ctx, out, name), want[k]):
                    assert torch.equal(a, b), (name, k)
        ctx.check()
