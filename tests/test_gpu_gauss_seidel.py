"""GPU: the Gauss-Seidel solve of the sparse J in one cluster launch, against the
row-by-row iteration in numpy (src/FESolver.cpp:561-601: checks after sweeps 1,
26, 51, ..., the sweep limit, rows with a tiny diagonal kept), from one CTA's
worth of rows to several, numbered by coordinate and at random, and a K that the
sparse solve does not take.

Tolerance: the iteration contracts, so the rounding of a sweep (a few 2^-53 of
sums of 15 terms) does not grow: 1e-12 relative after any number of sweeps."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import make_deck
import minipic_b200 as mp

pytestmark = pytest.mark.gpu


def sweeps(J, b, x, count):
    x = x.copy()
    for _ in range(count):
        for u in range(len(b)):
            if abs(J[u, u]) < 1e-12:
                continue
            nz = NZ[id(J)][u]
            x[u] = (b[u] - J[u, nz] @ x[nz] + J[u, u] * x[u]) / J[u, u]
    return x


NZ = {}


def run(ctx, b, limit):
    ctx.set_gs_max_sweeps(limit)
    ctx.build_j(mp.GAUSS_SEIDEL)
    J = ctx.fe_get("J")
    NZ[id(J)] = [np.nonzero(J[u])[0] for u in range(len(b))]
    try:
        st = ctx.solve_linear(mp.GAUSS_SEIDEL, mp.FP64, b=b)
        failed = False
    except mp.MpError as e:
        assert e.status == 5
        st, failed = None, True
    x, done = np.zeros_like(b), 0
    while done < limit:
        s = 1 if done == 0 else min(25, limit - done)
        x = sweeps(J, b, x, s)
        done += s
        if (done - 1) % 25 == 0 and np.linalg.norm(b - J @ x) / len(b) < 1e-4:
            assert not failed and st.linear_iterations == done - 1
            break
    else:
        assert failed
    y = ctx.fe_get("y")
    assert np.abs(y - x).max() <= 1e-12 * np.abs(x).max(), (limit, np.abs(y - x).max() / np.abs(x).max())


def context(dk, **kw):
    ctx = mp.Context(dk.mesh)
    ctx.fe_setup(**dk.fe_desc_arrays(-10.0), **kw)
    ctx.fe_set("d", np.random.default_rng(2).normal(0.0, 0.05, ctx.neq))
    return ctx


@pytest.mark.parametrize("n,sphere,limit", [(2, False, 1), (4, False, 40), (8, False, 27), (10, True, 51),
                                            (11, False, 2), (12, False, 26), (15, False, 3), (19, False, 2)])
def test_against_rows_in_order(tmp_path, n, sphere, limit):
    kd, path = make_deck(tmp_path, n, sphere=(50.0, 50.0, 50.0, 20.0) if sphere else None)
    ctx = context(mp.Deck.load(path))
    run(ctx, np.random.default_rng(n).normal(size=ctx.neq) * 0.1, limit)


def test_converges_at_a_check(tmp_path):
    kd, path = make_deck(tmp_path, 6)
    ctx = context(mp.Deck.load(path))
    run(ctx, np.random.default_rng(1).normal(size=ctx.neq) * 1e-3, 10000)


def test_random_numbering_and_kept_rows(tmp_path):
    """Random node numbers (long dependence levels), and rows whose diagonal is below 1e-12."""
    kd, path = make_deck(tmp_path, 7)
    p = np.random.default_rng(3).permutation(kd.n_nodes)
    pos = np.empty_like(kd.nodes_mm)
    pos[p] = kd.nodes_mm / 1000.0
    mesh = mp.Mesh.build(pos, p[kd.tets], p[kd.inlet_nodes], p[kd.inlet_tris], p[kd.wall_nodes])
    dk = mp.Deck(mp.Deck.load(path).params, mesh, kd.sphere_nodes)
    ctx = context(dk)
    run(ctx, np.random.default_rng(4).normal(size=ctx.neq) * 0.1, 27)
    ref = ctx
    K, F0 = ref.fe_get("K"), ref.fe_get("F0")
    fp = K - ref.fe_get("J")  # diagonal: the Boltzmann term
    for u in (0, 11, ref.neq - 1):
        K[u, u] = fp[u, u]
    ctx = context(dk, K=K, F0=F0)
    run(ctx, np.random.default_rng(5).normal(size=ctx.neq) * 0.1, 3)


def test_k_outside_the_pattern(tmp_path):
    """A coupling between unknowns of no common tet: the dense sweeps take it (they
    read J as symmetric)."""
    kd, path = make_deck(tmp_path, 6)
    dk = mp.Deck.load(path)
    ref = context(dk)
    K, F0 = ref.fe_get("K"), ref.fe_get("F0")
    far = np.argwhere(K[-1] == 0)[0, 0]
    K[-1, far] = K[far, -1] = 0.01 * K[0, 0]
    ctx = context(dk, K=K, F0=F0)
    run(ctx, np.random.default_rng(6).normal(size=ctx.neq) * 0.1, 26)
