"""Time steps past DT DX^2 / (2 RE) = 1/12, where the Crank-Nicolson coefficient
A = 1 - 12 q changes sign: still diagonally dominant systems (B = 10 + 24 q > 2 |A|), whose
decaying root is positive and grows towards 1 with q."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, C3D_MIXED, C3D_MIXED_IR, make_grid


def grid(n1m, n3m, q3, prec):
    """RE = 1/2, q in z as given, in x by (DX1 / DX3)^2 = (n1m / (2 n3m))^2."""
    g, _ = make_grid("small32", precision=prec, n1m=n1m, n2m=6, n3m=n3m, re=0.5)
    return g, 2 * g.re * q3 / g.arrays["dx3"] ** 2


def check(g, got, ref, prec, dt):
    # FP64: the parity tolerance of a step.  Mixed: the velocity bound of its step (its pressure
    # error is that of an FP32 divergence over DT, which these DT and RE make any size)
    tu = 1e-10 if prec == C3D_FP64 else 2e-5
    i, k = slice(1, g.n1m + 1), slice(1, g.n3m + 1)
    for c, j0 in ((0, 1), (1, 2), (2, 1)):
        a, b = (f[0][i, j0:g.n2m + 1, k, c] for f in (got, ref))
        assert np.all(np.isfinite(a)) and np.linalg.norm(a - b) < tu * np.linalg.norm(ref[0][i, 1:g.n2m + 1, k]), c
    if prec == C3D_FP64:   # the divergence's rounding over DT beside the parity tolerance
        a, b = (f[1][:g.n1m, :g.n2m, :g.n3m] for f in (got, ref))
        eps = np.finfo(float).eps * max(g.arrays["dx1"], g.arrays["dx3"]) / dt
        assert np.linalg.norm(a - b) < 1e-9 * np.linalg.norm(b) + eps * np.sqrt(b.size)


# q: A barely negative, |r| still within the warm-ups' reach, beyond it, and a long reach (the
# whole line many times over at q = 60: r = 0.88); rows in segments, whole warps and with idle
# lanes; lines that the joined form takes and one that it does not
@pytest.mark.gpu
@pytest.mark.parametrize("prec", [C3D_FP64, C3D_MIXED, C3D_MIXED_IR])
@pytest.mark.parametrize("n1m,n3m,q3", [(48, 32, 0.0834), (48, 32, 0.15), (48, 32, 0.25), (48, 32, 2.0), (48, 32, 60.0),
                                        (108, 48, 2.0), (256, 16, 0.5), (16, 1024, 0.5)])
def test_step_past_the_sign_change(oracle_mod, prec, n1m, n3m, q3):
    from compact3d_gb300 import build, lib
    build.build()
    g, dt = grid(n1m, n3m, q3, prec)
    orc = oracle_mod.Oracle(g)
    U, P, HH = ic.perturbed_laminar(g)
    orc.project(U)
    ch = lib.Channel(g, prec)
    ch.upload(U, P, HH)
    pg = pgo = (0.0, 0.0)
    for m in (1, 2):
        pgo = orc.getup(U, P, HH, m, dt, *pgo)
        pg = ch.step(m, dt, *pg)
    got = ch.download()
    ch.close()
    check(g, got, (U, P), prec, dt)


# roots within 1e-3 of 1 in x (1, 3 and 4 points a lane: segments, whole warps with and without
# idle lanes), which the ring's usual levels do not reach round
@pytest.mark.gpu
@pytest.mark.parametrize("n1m,batch", [(18, False), (24, False), (48, False), (108, False), (48, True)])
def test_roots_near_one(oracle_mod, n1m, batch):
    from compact3d_gb300 import build, lib
    build.build()
    q = 1e6
    g, dt = grid(n1m, 16, q * (32 / n1m) ** 2, C3D_FP64)
    orc = oracle_mod.Oracle(g)
    U, P, HH = ic.perturbed_laminar(g)
    orc.project(U)
    ch = lib.Batch([g]) if batch else lib.Channel(g)
    one = ch.channels[0] if batch else ch
    one.upload(U, P, HH)
    orc.getup(U, P, HH, 1, dt, 0.0, 0.0)
    if batch:
        ch.step(1, [dt], [0.0], [0.0])
    else:
        ch.step(1, dt, 0.0, 0.0)
    Ug = one.download()[0]
    ch.close()
    # the explicit terms' rounding, 12 q a term, which the solve passes on in its lowest modes
    tol = 100 * q * np.finfo(float).eps
    i, k = slice(1, g.n1m + 1), slice(1, g.n3m + 1)
    a, b = (f[i, 1:g.n2m + 1, k] for f in (Ug, U))
    assert np.linalg.norm(a - b) < tol * np.linalg.norm(b)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [C3D_FP64, C3D_MIXED])
def test_batch_past_the_sign_change(oracle_mod, prec):
    """The captured step follows DT from one side of the line to the other and back."""
    from compact3d_gb300 import build, lib
    build.build()
    ens = []
    for n1m, n3m in ((48, 32), (64, 48)):
        g, _ = grid(n1m, n3m, 1.0, prec)
        U, P, HH = ic.perturbed_laminar(g)
        orc = oracle_mod.Oracle(g)
        orc.project(U)
        ens.append((g, orc, U, P, HH))
    b = lib.Batch([e[0] for e in ens])
    for (g, orc, U, P, HH), ch in zip(ens, b.channels):
        ch.upload(U, P, HH)
    pb, pb3, po = [0.0, 0.0], [0.0, 0.0], [(0.0, 0.0)] * 2
    for m, q in enumerate((0.01, 0.6, 0.6, 0.01), 1):
        dts = [grid(e[0].n1m, e[0].n3m, q, prec)[1] for e in ens]
        pb, pb3 = b.step(m, dts, pb, pb3)
        po = [e[1].getup(e[2], e[3], e[4], m, dt, *p) for e, dt, p in zip(ens, dts, po)]
    for (g, orc, U, P, HH), ch in zip(ens, b.channels):
        check(g, ch.download(), (U, P), prec, dts[0])
    b.close()
