"""Mixed-state values whose low part is a denormal float, or that are denormal themselves,
come back from a download and a checkpoint as the state holds them."""
import numpy as np
import pytest

from compact3d_gb300.grid import C3D_MIXED, make_grid


@pytest.mark.gpu
def test_small_values_survive_download_and_checkpoint(tmp_path):
    from compact3d_gb300 import build, lib
    build.build()
    g, _ = make_grid("tiny16")
    rng = np.random.default_rng(2)
    U, P, HH = g.zeros_u(), g.zeros_p(), g.zeros_u()
    i, j, k = slice(1, g.n1m + 1), slice(2, g.n2m + 1), slice(1, g.n3m + 1)
    shape = (g.n1m, g.n2m - 1, g.n3m, 3)
    # 2^-74 (low parts from 2^-127 on) down to the smallest denormal float
    U[i, j, k] = rng.uniform(1, 2, shape) * 2.0 ** -rng.integers(74, 150, shape).astype(float) * rng.choice([-1, 1], shape)
    P[:g.n1m, 1:g.n2m, :g.n3m] = U[i, j, k, 0]
    ch = lib.Channel(g, C3D_MIXED)
    ch.upload(U, P, HH)

    def held(x):
        h = x.astype(np.float32)
        return h.astype(float) + (x - h.astype(float)).astype(np.float32).astype(float)

    Ug, Pg, _ = ch.download()
    assert np.array_equal(Ug[i, j, k], held(U[i, j, k]))
    assert np.array_equal(Pg[:g.n1m, 1:g.n2m, :g.n3m], held(P[:g.n1m, 1:g.n2m, :g.n3m]))
    f = str(tmp_path / "small.ckpt")
    ch.checkpoint_write(f, 3, 0.25, 0.0, 0.0)
    ch.close()
    ch = lib.Channel(g, C3D_MIXED)
    ch.checkpoint_read(f)
    U2, P2, _ = ch.download()
    ch.close()
    assert np.array_equal(U2[i, j, k], Ug[i, j, k])
    assert np.array_equal(P2[:g.n1m, 1:g.n2m, :g.n3m], Pg[:g.n1m, 1:g.n2m, :g.n3m])
