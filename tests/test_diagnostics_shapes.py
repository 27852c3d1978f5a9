"""Per-step diagnostics (c3d_diagnose) at the edges of their kernels' shapes."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, C3D_MIXED, make_grid


def test_float_to_double_bits():
    """numpy model of f2d (c3d_kern.cuh): exact for every float but denormals, which become zero."""
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.integers(0, 1 << 32, 200000, dtype=np.uint64).astype(np.uint32),
                        np.array([0, 1 << 31, 0x7f800000, 0xff800000, 0x7fc00000, 0x00800000, 0x7f7fffff], np.uint32)])
    e = x & 0x7f800000
    hi = ((x & 0x7fffffff) >> 3) + np.uint32(0x38000000)
    lo = x << np.uint32(29)
    hi = np.where(e == 0x7f800000, hi + np.uint32(0x38000000), hi)
    hi, lo = np.where(e == 0, 0, hi), np.where(e == 0, 0, lo)
    hi = hi | (x & np.uint32(0x80000000))
    got = ((hi.astype(np.uint64) << np.uint64(32)) | lo).view(np.float64)
    with np.errstate(invalid="ignore"):   # signalling NaNs
        ref = x.view(np.float32).astype(np.float64)
    ref = np.where(np.abs(ref) < 2.0 ** -126, np.copysign(0.0, ref), ref)
    assert np.array_equal(got, ref, equal_nan=True)


# one block of sums and many; joined z lines of 8, 12 and 16 points, a line too long for a
# block; rows with idle lanes
@pytest.mark.gpu
@pytest.mark.parametrize("prec", [C3D_FP64, C3D_MIXED])
@pytest.mark.parametrize("shape", [(16, 4, 16), (36, 9, 48), (108, 20, 144), (24, 5, 768), (16, 4, 1024), (96, 64, 128)])
def test_diagnostics_match_oracle(oracle_mod, prec, shape):
    from compact3d_gb300 import build, lib
    build.build()
    g, dt = make_grid("small32", n1m=shape[0], n2m=shape[1], n3m=shape[2])
    orc = oracle_mod.Oracle(g)
    U, P, HH = ic.perturbed_laminar(g, amp=0.3)      # not projected: the divergence is not rounding
    ch = lib.Channel(g, prec)
    ch.upload(U, P, HH)
    U, _, _ = ch.download()                          # what the state holds, with its ghost columns
    for _ in range(2):
        d = ch.diagnose()
        f1, f3 = orc.chkmf(U)
        assert not d["nonfinite"]
        # sums of n terms in another order, solves truncated below rounding
        assert abs(d["divmax"] - orc.divcheck(U)) <= 1e-11 * orc.divcheck(U)
        assert abs(d["cflm"] - orc.cfl(U)) <= 1e-13 * orc.cfl(U)
        assert abs(d["flow1"] - f1) <= 1e-12 * abs(f1) and abs(d["flow3"] - f3) <= 1e-12 * abs(f1)
        w = np.asarray(orc.wallss(U))
        assert np.max(np.abs(d["wsm"] - w)) <= 1e-11 * np.max(np.abs(w))
    U[3, 2, 4, 0] = np.nan
    ch.upload(U, P, HH)
    assert ch.diagnose()["nonfinite"]
    ch.close()
