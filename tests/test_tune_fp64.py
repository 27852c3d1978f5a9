"""The tuner leaves the knobs that FP64 does not read (z segment lengths, staged xA rows, row
lanes) at their values instead of choosing between equal kernels."""
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, make_grid

UNREAD = [f"z_segment_z{c}" for c in "ABCDE"] + ["x_stage_xA", "x_row_lanes"]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(64, 12, 32), (96, 10, 64)])
def test_fp64_autotune_keeps_unread_knobs(shape):
    from compact3d_gb300 import build, lib
    build.build()
    g, _ = make_grid("small32", n1m=shape[0], n2m=shape[1], n3m=shape[2])
    ch = lib.Channel(g, C3D_FP64)
    ch.upload(*ic.perturbed_laminar(g))
    before = ch.get_schedule()
    after = ch.autotune()
    assert {k: after[k] for k in UNREAD} == {k: before[k] for k in UNREAD}
    ch.close()
