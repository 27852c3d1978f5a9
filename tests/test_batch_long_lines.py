"""Work-list batches with z lines whose FFT tile of 8 kx columns would not fit in shared
memory, beside a channel of short lines: the tile narrows for the long one alone."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, C3D_MIXED, make_grid


# FP64: 256 KB at 8 columns (tile 4), on lines whose z passes run the warm-up form too, and
# 4 columns too wide (tile 2); mixed: 288 KB at 8 columns
@pytest.mark.gpu
@pytest.mark.parametrize("prec,n3m", [(C3D_FP64, 1024), (C3D_FP64, 2304), (C3D_MIXED, 2304)])
def test_long_z_lines_in_a_batch(oracle_mod, prec, n3m):
    from compact3d_gb300 import build, lib
    build.build()
    ens = []
    for n3 in (n3m, 48):
        g, dt = make_grid("small32", precision=prec, n1m=18, n2m=5, n3m=n3)
        U, P, HH = ic.perturbed_laminar(g)
        orc = oracle_mod.Oracle(g)
        orc.project(U)
        ens.append((g, dt, orc, U, P, HH))
    b = lib.Batch([e[0] for e in ens])
    assert b.get_form() == "worklist"
    for (g, dt, orc, U, P, HH), ch in zip(ens, b.channels):
        ch.upload(U, P, HH)
    pb, pb3, po = [0.0, 0.0], [0.0, 0.0], [(0.0, 0.0)] * 2
    for m in (1, 2):
        pb, pb3 = b.step(m, [e[1] for e in ens], pb, pb3)
        po = [e[2].getup(e[3], e[4], e[5], m, e[1], *p) for e, p in zip(ens, po)]
    tu, tp = (1e-10, 1e-9) if prec == C3D_FP64 else (2e-5, 1e-3)     # as for one channel
    for (g, dt, orc, U, P, HH), ch in zip(ens, b.channels):
        Ug, Pg, _ = ch.download()
        for c, j0 in ((0, 1), (1, 2), (2, 1)):
            x, y = (f[1:19, j0:6, 1:g.n3m + 1, c] for f in (Ug, U))
            assert np.linalg.norm(x - y) / np.linalg.norm(y) < tu, (g.n3m, c)
        x, y = (f[:18, :5, :g.n3m] for f in (Pg, P))
        assert np.linalg.norm(x - y) / np.linalg.norm(y) < tp, g.n3m
    b.close()
