"""The wall-normal factor's form: the default of a grid shows in its schedule, and a form that
a schedule names is the one that is set."""
import pytest

from compact3d_gb300.grid import C3D_FP64, C3D_MIXED, make_grid


# just below and at the size from which mixed grids default to tiles of 64 columns; FP64 keeps
# the register form
@pytest.mark.gpu
@pytest.mark.parametrize("prec,shape,default", [(C3D_MIXED, (64, 16, 64), 0), (C3D_MIXED, (384, 172, 512), 64),
                                                (C3D_MIXED, (256, 255, 512), 0), (C3D_FP64, (384, 172, 512), 0)])
def test_default_form_and_explicit_choice(prec, shape, default):
    from compact3d_gb300 import build, lib
    build.build()
    g, _ = make_grid("small32", n1m=shape[0], n2m=shape[1], n3m=shape[2])
    ch = lib.Channel(g, prec)
    s = ch.get_schedule()
    assert s["ycn_tile"] == default
    for t in (0, 32, 64):
        ch.set_schedule(dict(s, ycn_tile=t))
        assert ch.get_schedule()["ycn_tile"] == t
    ch.close()
