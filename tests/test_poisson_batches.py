"""The Poisson sweeps along y in batches of 8 planes with two sets of registers (pz_sweeps):
every way the planes can end, against the oracle."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, C3D_MIXED, make_grid


@pytest.mark.gpu
@pytest.mark.parametrize("n2m", [4, 7, 8, 9, 15, 16, 17, 18, 24, 25, 33])
@pytest.mark.parametrize("prec", [C3D_FP64, C3D_MIXED])
def test_poisson_matches_oracle(oracle_mod, n2m, prec):
    from compact3d_gb300 import build, lib
    build.build()
    g, dt = make_grid("small32", n1m=16, n2m=n2m, n3m=16)
    orc = oracle_mod.Oracle(g)
    U, P, HH = ic.perturbed_laminar(g)
    orc.project(U)
    ch = lib.Channel(g, prec)
    ch.upload(U, P, HH)
    pg = pgo = (0.0, 0.0)
    for m in (1, 2):
        pgo = orc.getup(U, P, HH, m, dt, *pgo)
        pg = ch.step(m, dt, *pg)
    Ug, Pg, _ = ch.download()
    ch.close()
    # FP64: rounding; mixed: the bound of the mixed form, and DP from FP32 right-hand sides over DT
    tu, tp = (1e-10, 1e-9) if prec == C3D_FP64 else (2e-5, 1e-3)
    for c, j0 in ((0, 1), (1, 2), (2, 1)):
        a, b = (f[1:17, j0:n2m + 1, 1:17, c] for f in (Ug, U))
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < tu, c
    assert np.linalg.norm(Pg[:16, :n2m, :16] - P[:16, :n2m, :16]) / np.linalg.norm(P[:16, :n2m, :16]) < tp
