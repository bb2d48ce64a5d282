"""The reverse mode's field gradient where a block's threads are odd in number
(FP32: nvx / 4 thread rows of as many columns as 512 threads hold), so that the
sums behind its ring of rows need padding: against the FP64 CPU adjoint."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import IC_LANDAU_SUM, Restatement

pytestmark = pytest.mark.gpu


# nvx, columns per block asked for ("": the default, 17 at nvx = 116, 15 at 132, 13 at 148).
@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("nvx,columns", [(116, ""), (132, ""), (148, ""), (128, ""), (12, "7"), (20, "1"), (12, "")])
def test_step_adjoint(pkg, cuda, monkeypatch, nvx, columns, dtype):
    torch = cuda
    if columns:
        monkeypatch.setenv("VLP4D_VGRAD_CW", columns)
    n = (8, 9, nvx, 10)
    L = 4 * np.pi
    dom = pkg.Domain(list(n), [0.0, 0.0, -6.0, -6.0], [L, L, 6.0, 6.0], 0.1, 2, 110)
    ora = Restatement(dom.nxmax, dom.min_phy, dom.max_phy, dom.dt, dom.idcase)
    f1 = ora.step(ora.init_case(IC_LANDAU_SUM, 0.05, 0.5))
    lam = np.random.default_rng(nvx).normal(size=ora.shape4)
    with pkg.Context(dom, dtype) as ctx, pkg.Adjoint(ctx, 1, 1) as adj:
        out = ctx.empty_f()
        dev = lambda x: torch.from_numpy(x).to(ctx.torch_dtype).cuda()  # noqa: E731
        adj.step_adjoint(dev(f1), dev(lam), out)
        ctx.check()
        got = out.double().cpu().numpy()
    ref = ora.step_adjoint(f1, lam)
    # FP32: some sixty roundings of 6e-8 in sums of a magnitude of max|ref|.
    tol = 1e-11 if dtype == "f64" else 60 * 6e-8
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
