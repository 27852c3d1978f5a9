"""SGSDY's tiled filter and sums on planes that a tile of 32 x 16 points overhangs, divides
and wraps: one FP64 step against the oracle."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, make_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 8, 16), (18, 8, 48), (36, 9, 16), (64, 8, 32), (108, 8, 16)])
def test_sgsdy_step_matches_oracle(oracle_mod, shape):
    from compact3d_gb300 import build, lib
    build.build()
    g, dt = make_grid("les32dy", n1m=shape[0], n2m=shape[1], n3m=shape[2])
    orc = oracle_mod.Oracle(g)
    U, P, HH = ic.loglaw(g, 2000.0)
    orc.project(U)
    ch = lib.Channel(g, C3D_FP64)
    ch.upload(U, P, HH)
    S = g.zeros_s()
    pg = pgo = (0.0, 0.0)
    for m in (1, 2):
        pgo = orc.getup(U, P, HH, m, dt, *pgo, sgsvis=S)
        pg = ch.step(m, dt, *pg)
    Ug, _, _ = ch.download()
    i, j, k = slice(1, shape[0] + 1), slice(1, shape[1] + 1), slice(1, shape[2] + 1)
    Sg = ch.download_sgsvis()
    ch.close()
    # nu = C |S| with C a ratio of sums whose terms cancel (L:M); the parity tolerance of a step
    assert np.linalg.norm(Sg[i, j, k] - S[i, j, k]) <= 1e-9 * np.linalg.norm(S[i, j, k])
    for c in range(3):
        a, b = Ug[i, j, k, c], U[i, j, k, c]
        assert np.linalg.norm(a - b) <= 1e-10 * np.linalg.norm(b), c
