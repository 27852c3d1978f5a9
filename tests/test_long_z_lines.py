"""z lines whose widest FFT tile would not fit in shared memory: the tile narrows."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, make_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n3m,tile", [(512, 8), (512, 16), (1024, 8)])
def test_long_z_lines_fp64(oracle_mod, n3m, tile):
    from compact3d_gb300 import build, lib
    build.build()
    g, dt = make_grid("small32", n1m=16, n2m=5, n3m=n3m)
    orc = oracle_mod.Oracle(g)
    U, P, HH = ic.perturbed_laminar(g)
    orc.project(U)
    ch = lib.Channel(g, C3D_FP64)
    ch.upload(U, P, HH)
    ch.set_schedule(dict(ch.get_schedule(), fft_z_tile=tile))
    orc.getup(U, P, HH, 1, dt, 0.0, 0.0)
    ch.step(1, dt, 0.0, 0.0)
    Ug, Pg, _ = ch.download()
    ch.close()
    for c, j0 in ((0, 1), (1, 2), (2, 1)):
        a, b = (f[1:17, j0:6, 1:n3m + 1, c] for f in (Ug, U))
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < 1e-10, c
