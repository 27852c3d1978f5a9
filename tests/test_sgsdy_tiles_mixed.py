"""SGSDY's tiled filter and sums in the mixed form, whose filter divides where FP64 scales: two
steps against the oracle on planes that a tile of 32 x 16 points overhangs, divides and wraps."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_MIXED, make_grid


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(16, 8, 16), (18, 8, 48), (36, 9, 16), (64, 8, 32), (108, 8, 16)])
def test_mixed_sgsdy_step_matches_oracle(oracle_mod, shape):
    from compact3d_gb300 import build, lib
    build.build()
    g, dt = make_grid("les32dy", n1m=shape[0], n2m=shape[1], n3m=shape[2])
    orc = oracle_mod.Oracle(g)
    U, P, HH = ic.loglaw(g, 2000.0)
    orc.project(U)
    ch = lib.Channel(g, C3D_MIXED)
    ch.upload(U, P, HH)
    S = g.zeros_s()
    pg = pgo = (0.0, 0.0)
    for m in (1, 2):
        pgo = orc.getup(U, P, HH, m, dt, *pgo, sgsvis=S)
        pg = ch.step(m, dt, *pg)
    Ug, _, _ = ch.download()
    Sg = ch.download_sgsvis()
    ch.close()
    i, j, k = slice(1, shape[0] + 1), slice(1, shape[1] + 1), slice(1, shape[2] + 1)
    # the tolerances of the mixed LES form against FP64: nu = C |S| with C a ratio of sums of
    # cancelling FP32 products
    assert np.linalg.norm(Sg[i, j, k] - S[i, j, k]) <= 1e-3 * np.linalg.norm(S[i, j, k])
    assert np.linalg.norm(Ug[i, j, k] - U[i, j, k]) <= 1e-4 * np.linalg.norm(U[i, j, k])
