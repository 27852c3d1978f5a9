"""The bulk-copy ring exists in the mixed form alone: in FP64 its knob changes nothing, so a
schedule that names it takes the same kernels, bit for bit."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, make_grid


@pytest.mark.gpu
@pytest.mark.parametrize("n1m", [64, 96, 108])
def test_bulk_stages_do_nothing_in_fp64(n1m):
    from compact3d_gb300 import build, lib
    build.build()
    g, dt = make_grid("small32", n1m=n1m, n2m=8, n3m=32)
    U, P, HH = ic.perturbed_laminar(g)
    out = []
    for stages in (0, 2, 3):
        ch = lib.Channel(g, C3D_FP64)
        ch.upload(U, P, HH)
        ch.set_schedule(dict(ch.get_schedule(), x_bulk_stages=stages))
        pg = (0.0, 0.0)
        for m in (1, 2):
            pg = ch.step(m, dt, *pg)
        out.append(ch.download())
        ch.close()
    for r in out[1:]:
        for a, b in zip(r, out[0]):
            assert np.array_equal(a, b)
