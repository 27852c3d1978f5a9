"""Joined z segments (zjoin in c3d_dev.cuh): the state entering a segment comes from the
K = ceil(M / L) segments before it (after it, backward), each weighted by r^L per segment
crossed, M the length after which |r|^M is below the precision's rounding unit."""
import numpy as np
import pytest

from compact3d_gb300 import ic
from compact3d_gb300.grid import C3D_FP64, C3D_MIXED, make_grid


def join(d, L, M, r):
    """numpy model of zjoin on one line: B(F(d)) by segments."""
    n = len(d)
    nseg, K = n // L, -(-M // L)
    x = d.reshape(nseg, L).copy()

    def sweep(x, order, step):
        y = np.zeros(nseg)
        for t in order:
            y = x[:, t] + r * y
        seg = np.arange(nseg)
        c = y[(seg - step * K) % nseg]
        for k in range(K - 1, 0, -1):
            c = y[(seg - step * k) % nseg] + r ** L * c
        for t in order:
            c = x[:, t] + r * c
            x[:, t] = c

    sweep(x, range(L), 1)
    sweep(x, range(L - 1, -1, -1), -1)
    return x.reshape(-1)


@pytest.mark.parametrize("n3m", [16, 32, 48, 96, 144, 288, 512, 768])
@pytest.mark.parametrize("b", [6.0, 10.0, 22.0])
def test_join_solves_the_cyclic_system(n3m, b):
    """(1, b, 1) cyclic: s B(F(d)) against the dense solve, every segment length that divides
    the line, lines of fewer segments than a carry spans among them (N3M = 16, L = 8)."""
    r = -2.0 / (b + np.sqrt(b * b - 4.0))
    d = np.random.default_rng(n3m).normal(size=n3m)
    A = b * np.eye(n3m) + np.eye(n3m, k=1) + np.eye(n3m, k=-1)
    A[0, -1] = A[-1, 0] = 1.0
    ref = np.linalg.solve(A, d)
    for L in (8, 12, 16):
        if n3m % L == 0:
            x = -r * join(d, L, 23, r)
            # truncation |r|^23 <= 3e-18 and the rounding of 2 n3m multiply-adds that decay by |r|
            assert np.max(np.abs(x - ref)) <= 20 * np.finfo(float).eps * np.max(np.abs(ref)), (L, n3m, b)


@pytest.fixture(scope="module")
def libc3d():
    from compact3d_gb300 import build, lib
    build.build()
    lib.load()
    return lib


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


# N3M: 2 segments of 8 (a carry of 3 segments goes round the line), segments of 12, of 8 at
# the most segments a block holds (64), of 16 (48 segments), and a line too long for a block
# (the warm-up form); N1M and N2M leave the last block part of its columns and put columns of
# two planes in one block
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(18, 9, 16), (36, 11, 48), (32, 7, 144), (16, 5, 512), (24, 5, 768), (16, 4, 1024)])
def test_joined_fp64_step_matches_oracle(libc3d, oracle_mod, shape):
    n1m, n2m, n3m = shape
    g, dt = make_grid("small32", n1m=n1m, n2m=n2m, n3m=n3m)
    orc = oracle_mod.Oracle(g)
    U, P, HH = ic.perturbed_laminar(g)
    orc.project(U)
    ch = libc3d.Channel(g, C3D_FP64)
    ch.upload(U, P, HH)
    pg = pgo = (0.0, 0.0)
    for m in (1, 2):
        pgo = orc.getup(U, P, HH, m, dt, *pgo)
        pg = ch.step(m, dt, *pg)
    Ug, Pg, HHg = ch.download()
    ch.close()
    i, k = slice(1, n1m + 1), slice(1, n3m + 1)
    for c, j0 in ((0, 1), (1, 2), (2, 1)):
        assert rel(Ug[i, j0:n2m + 1, k, c], U[i, j0:n2m + 1, k, c]) < 1e-10, c
        assert rel(HHg[i, j0:n2m + 1, k, c], HH[i, j0:n2m + 1, k, c]) < 1e-9, c
    assert rel(Pg[:n1m, :n2m, :n3m], P[:n1m, :n2m, :n3m]) < 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(18, 9, 16), (36, 11, 48), (108, 9, 144), (16, 5, 288)])
def test_joined_mixed_step_close_to_segments(libc3d, shape):
    """Schedule 0 of the mixed form on rows that are not a multiple of 32 points: three steps
    agree with the warm-up segments' to FP32 rounding of the increments."""
    n1m, n2m, n3m = shape
    g, dt = make_grid("small32", n1m=n1m, n2m=n2m, n3m=n3m)
    U, P, HH = ic.perturbed_laminar(g)
    res = []
    for zl in (16, 0):
        ch = libc3d.Channel(g, C3D_MIXED)
        ch.upload(U, P, HH)
        ch.set_schedule(dict(ch.get_schedule(), **{f"z_segment_z{c}": zl for c in "ABCDE"}))
        for m in (1, 2, 3):
            ch.step(m, dt, 0.0, 0.0)
        res.append(ch.download()[0])
        ch.close()
    for c, j0 in ((0, 1), (1, 2), (2, 1)):
        a, b = (r[1:n1m + 1, j0:n2m + 1, 1:n3m + 1, c] for r in res)
        assert rel(b, a) < 1e-5, (c, rel(b, a))
