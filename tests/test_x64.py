"""The FP64 x passes: rows in segments by N1M, folded factors, and the Crank-Nicolson factors
of x and z as partial fractions (xa64, ab2_cnx, cn_factors)."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, make_grid


@pytest.mark.parametrize("q", [0.0, 1e-7, 1e-4, 3e-3, 0.02])
@pytest.mark.parametrize("n", [16, 54])
def test_cn_partial_fractions(q, n):
    """(1, 10, 1) x / (A, B, A) against x / A + k z / (1, B/A, 1) x: A = 1 - 12 q, B = 10 + 24 q."""
    A, B = 1.0 - 12 * q, 10.0 + 24 * q
    shift = np.roll(np.eye(n), 1, 0) + np.roll(np.eye(n), -1, 0)
    x = np.random.default_rng(n).normal(size=n)
    ref = np.linalg.solve(A * shift + B * np.eye(n), shift @ x + 10 * x)
    beta = B / A
    r = -2.0 / (beta + np.sqrt(beta * beta - 4.0))
    assert abs(-r * (10 - beta)) <= 0.5 and A > 0.5          # the range the kernels take this form in
    got = (x + (10 - beta) * np.linalg.solve(shift + beta * np.eye(n), x)) / A
    # two terms of the result's size, and the dense solves' own rounding
    assert np.max(np.abs(got - ref)) <= 40 * np.finfo(float).eps * np.max(np.abs(ref))


CASES = [(n, {}, {}) for n in (24, 48, 64, 96, 128, 192)]
CASES += [(n, {"x_split_xA": 1, "x_stage_xA": 1}, {}) for n in (24, 64, 192)]      # staged rows: a warp per row
CASES += [(n, {"fft_x_plan": 3, "x_split_xA": 1}, {}) for n in (64, 192)]          # the register row FFT
# k past 1/2 in z or x (A still positive): the stencil
CASES += [(48, {"x_rows_per_block": 2}, {"re": 20.0, "dt": 0.023}), (108, {"x_rows_per_block": 2}, {"re": 20.0, "dt": 0.008})]
CASES += [(64, {}, {"n3m": 768})]                                                   # lines zC joins by 16
CASES += [(16, {}, {"n3m": 1024})]                                                  # lines it does not join


@pytest.mark.gpu
@pytest.mark.parametrize("n1m,knobs,opt", CASES)
def test_fp64_rows_match_oracle(oracle_mod, n1m, knobs, opt):
    from compact3d_gb300 import build, lib
    build.build()
    kw = {"re": opt["re"]} if "re" in opt else {}
    n3m = opt.get("n3m", 32)
    g, dt = make_grid("small32", n1m=n1m, n2m=5, n3m=n3m, **kw)
    dt = opt.get("dt", dt)
    orc = oracle_mod.Oracle(g)
    U, P, HH = ic.perturbed_laminar(g)
    orc.project(U)
    ch = lib.Channel(g, C3D_FP64)
    ch.upload(U, P, HH)
    if knobs:
        ch.set_schedule(dict(ch.get_schedule(), **knobs))
    pg = pgo = (0.0, 0.0)
    for m in (1, 2):
        pgo = orc.getup(U, P, HH, m, dt, *pgo)
        pg = ch.step(m, dt, *pg)
    Ug, Pg, _ = ch.download()
    ch.close()
    for c, j0 in ((0, 1), (1, 2), (2, 1)):
        a, b = (f[1:n1m + 1, j0:6, 1:n3m + 1, c] for f in (Ug, U))
        assert np.linalg.norm(a - b) / np.linalg.norm(b) < 1e-10, c
    assert np.linalg.norm(Pg[:n1m, :5, :n3m] - P[:n1m, :5, :n3m]) / np.linalg.norm(P[:n1m, :5, :n3m]) < 1e-9
