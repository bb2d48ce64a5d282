"""Ensemble members whose plane sides are primes, squares of primes, the
largest allowed and shorter than any factor, against single runs through the
cuFFT field solve: the in-kernel solve's two-factor transforms, its joined
inverse of Ex and Ey and their Nyquist modes (tolerances of the other
ensemble-against-single-run tests)."""
from __future__ import annotations

import numpy as np
import pytest

from test_ensemble_gpu import _members, _single_run

pytestmark = pytest.mark.gpu

DIMS = [(17, 13, 8, 9), (64, 64, 8, 8), (37, 10, 9, 8), (15, 49, 8, 8), (2, 6, 8, 70), (63, 64, 8, 7), (6, 3, 12, 8)]


def test_members_match_single_runs(pkg, cuda, monkeypatch):
    torch = cuda
    nsteps = 4
    members = _members(pkg, DIMS)
    monkeypatch.setenv("VLP4D_FIELD", "cufft")
    with pkg.Ensemble(members, nsteps) as ens:
        ens.run()
        ens.check()
        for i, m in enumerate(members):
            f, nrj = ens.read(i)
            f_ref, nrj_ref = _single_run(pkg, torch, m, nsteps)
            assert float((f - f_ref).abs().max()) <= 2e-6 * float(f_ref.abs().max()), i
            assert np.abs(nrj - nrj_ref).max() < 1e-6, (i, nrj, nrj_ref)
