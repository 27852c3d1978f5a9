"""ENERGY's statistics at the edges of the marching kernels' shapes: rows shorter than a
warp's 30 columns, just past one and two groups of them, odd half rows, chunks of k that
do not divide N3M, one and many planes."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, C3D_MIXED, make_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [C3D_FP64, C3D_MIXED])
@pytest.mark.parametrize("shape", [(16, 4, 16), (32, 5, 48), (54, 7, 16), (64, 40, 32), (108, 9, 144), (384, 4, 16)])
def test_statistics_match_oracle(oracle_mod, prec, shape):
    from compact3d_gb300 import build, lib
    build.build()
    g, dt = make_grid("small32", n1m=shape[0], n2m=shape[1], n3m=shape[2])
    orc = oracle_mod.Oracle(g)
    U, P, _ = ic.perturbed_laminar(g, amp=0.3)
    P[:g.n1m, :g.n2m, :g.n3m] = np.random.default_rng(1).normal(size=(g.n1m, g.n2m, g.n3m))
    ch = lib.Channel(g, prec)
    ch.upload(U, P, g.zeros_u())
    U, P, _ = ch.download()        # the state's values
    s, ref = ch.plane_stats(), orc.plane_stats(U, P)
    # FP64 sums of up to N1M N3M terms in another order; a column that sums to nothing is
    # measured against the terms it sums (the unit of its square)
    scale = np.maximum(np.linalg.norm(ref, axis=0), 0.1)
    assert np.max(np.linalg.norm(s - ref, axis=0) / scale) < 1e-12
    sp = ch.plane_spectra()
    rs = orc.plane_spectra(U)
    for q, (k, tol) in enumerate((("xspec", 1e-12), ("zspec", 1e-12), ("rxx", 1e-9), ("rzz", 1e-9), ("rxy", 1e-9))):
        r = rs[k] if isinstance(rs, dict) else rs[q]
        assert np.linalg.norm(sp[k] - r) <= tol * np.linalg.norm(r), k
    vmo = np.asfortranarray(0.01 + ref[:, :3])
    assert np.linalg.norm(ch.plane_spectra(vmo)["zspec"] - (orc.plane_spectra(U, vmo)["zspec"] if isinstance(rs, dict)
                          else orc.plane_spectra(U, vmo)[1])) <= 1e-12 * np.linalg.norm(rs["zspec"] if isinstance(rs, dict) else rs[1])
    q, rq = ch.plane_quadrants(), orc.plane_quadrants(U)
    assert np.array_equal(q[:, 4:], rq[:, 4:]) and np.linalg.norm(q - rq) <= 1e-12 * np.linalg.norm(rq)
    ch.close()
