"""FP64 line solves along x by ring doubling (xsolve_ring in c3d_dev.cuh)."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, make_grid

# every lane-chunk shape: whole warps and segments (W = 8, 16), full and with idle lanes
ROWS = [(16, 1), (18, 1), (24, 1), (32, 1), (36, 2), (48, 2), (54, 2), (64, 2), (72, 3), (96, 3), (108, 4), (128, 4),
        (162, 6), (192, 6), (256, 8), (384, 12), (48, 6), (64, 8), (96, 12), (128, 8)]


def ring(e, m, step):
    P, off, levels = len(e), 1, 0
    lane = np.arange(P)
    while levels < 12 and abs(m) >= 2.0 ** -56:
        e = e + m * e[(lane - step * off) % P]
        m, off, levels = m * m, (2 * off) % P, levels + 1
    return e[(lane - step) % P]


@pytest.mark.parametrize("n,C", ROWS)
@pytest.mark.parametrize("b", [6.0, 10.0, 22.0, 2.5])
def test_ring_solves_the_cyclic_system(n, C, b):
    """Against the dense solve of the cyclic (1, b, 1) system; b = 2.5 (|r| = 1/2) runs the
    doubling round the ring on short rows."""
    r = -2.0 / (b + np.sqrt(b * b - 4.0))
    d = np.random.default_rng(n).normal(size=n)
    x = d.reshape(n // C, C).copy()
    for order, step in ((range(C), 1), (range(C - 1, -1, -1), -1)):
        e = np.zeros(n // C)
        for t in order:
            e = x[:, t] + r * e
        y = ring(e, r ** C, step)
        for t in order:
            y = x[:, t] + r * y
            x[:, t] = y
    A = b * np.eye(n) + np.eye(n, k=1) + np.eye(n, k=-1)
    A[0, -1] = A[-1, 0] = 1.0
    ref = np.linalg.solve(A, d)
    # rounding of four sweeps whose errors decay by |r| per point, and the dense solve's own
    assert np.max(np.abs(-r * x.reshape(-1) - ref)) <= 40 * np.finfo(float).eps * np.max(np.abs(ref))


@pytest.mark.gpu
@pytest.mark.parametrize("n1m", [16, 18, 24, 32, 36, 54, 72, 96, 108, 162, 256])
@pytest.mark.parametrize("split", [0, 1])
def test_fp64_step_matches_oracle_on_every_row_shape(oracle_mod, n1m, split):
    from compact3d_gb300 import build, lib
    build.build()
    g, dt = make_grid("small32", n1m=n1m, n2m=6, n3m=16)
    orc = oracle_mod.Oracle(g)
    U, P, HH = ic.perturbed_laminar(g)
    orc.project(U)
    ch = lib.Channel(g, C3D_FP64)
    ch.upload(U, P, HH)
    ch.set_schedule(dict(ch.get_schedule(), x_split_xA=split))
    pg = pgo = (0.0, 0.0)
    for m in (1, 2):
        pgo = orc.getup(U, P, HH, m, dt, *pgo)
        pg = ch.step(m, dt, *pg)
    Ug, Pg, _ = ch.download()
    ch.close()
    for c, j0 in ((0, 1), (1, 2), (2, 1)):
        a, b = (f[1:n1m + 1, j0:7, 1:17, c] for f in (Ug, U))
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < 1e-10, c
    assert np.linalg.norm(Pg[:n1m, :6, :16] - P[:n1m, :6, :16]) / np.linalg.norm(P[:n1m, :6, :16]) < 1e-9
