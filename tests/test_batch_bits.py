"""The mixed convective terms of a channel in an ensemble are those of the channel alone under
the same schedule, bit for bit, whatever the segment length of zB."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_MIXED, make_grid


@pytest.mark.gpu
@pytest.mark.parametrize("zb", [8, 16, 32])
def test_worklist_terms_have_the_single_channels_bits(zb):
    from compact3d_gb300 import build, lib
    build.build()
    zseg = (8, zb, 16, 16, 8)
    ens = [make_grid("channel64", precision=C3D_MIXED, n1m=n1, n2m=n2, n3m=n3)
           for n1, n2, n3 in ((48, 16, 64), (96, 12, 96), (128, 9, 128))]
    b = lib.Batch([g for g, _ in ens])
    b.set_z_segments(zseg)
    singles = []
    for (g, dt), ch in zip(ens, b.channels):
        U, P, HH = ic.perturbed_laminar(g)
        ch.upload(U, P, HH)
        s = lib.Channel(g)
        s.upload(U, P, HH)
        sched = dict(s.get_schedule(), x_rows_per_block=2, fft_z_tile=0, z_split_zA=1, x_split_xA=1,
                     fft_x_plan=3 if g.n1m % 64 == 0 else 0, x_row_lanes=16 if g.n1m == 128 else 8)
        sched.update({f"z_segment_z{c}": z for c, z in zip("ABCDE", zseg)})
        s.set_schedule(sched)
        singles.append(s)
    b.step(1, [dt for _, dt in ens], [0.0] * 3, [0.0] * 3)
    for (g, dt), ch, s in zip(ens, b.channels, singles):
        s.step(1, dt, 0.0, 0.0)
        in_batch, alone = ch.download()[2], s.download()[2]
        assert np.array_equal(in_batch, alone)
        s.close()
    b.close()
