"""GPU: SPARSE_CG's multilevel conjugate gradients, against the J of the dense
storage, from one block with a part of a cell's rows to some tens of blocks and
three levels; in both storages; in a thin, randomly numbered mesh; with a
Boltzmann term that outweighs K; and what the solver refuses.

Tolerance: the solver stops at ||b - J y|| <= 1e-12 ||b|| by its own rounding, so
numpy's residual is within that and the rounding of both row sums of at most 20
terms, 2 * 20 * 2^-53 || |J| |y| ||."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import make_deck
import minipic_b200 as mp

pytestmark = pytest.mark.gpu


def context(dk, storage=mp.FE_DENSE, **kw):
    ctx = mp.Context(dk.mesh)
    ctx.set_fe_storage(storage)
    ctx.fe_setup(**dk.fe_desc_arrays(None), **kw)
    return ctx


def solve(ctx, d, b):
    ctx.fe_set("d", d)
    ctx.build_j(mp.SPARSE_CG)
    st = ctx.solve_linear(mp.SPARSE_CG, mp.FP64, b=b)
    return ctx.fe_get("y"), st


def dense_j(ctx, d):
    ctx.fe_set("d", d)
    ctx.build_j(mp.LAPACK)
    return ctx.fe_get("J")


def holds(J, y, b):
    bound = 1e-12 * np.linalg.norm(b) + 40 * 2.0 ** -53 * np.linalg.norm(np.abs(J) @ np.abs(y))
    return np.linalg.norm(b - J @ y) <= bound


def by_diagonal(J, b):
    """Iterations of conjugate gradients with J's diagonal."""
    J, b = -J, -b
    r, D = b.copy(), np.diag(J)
    z = r / D
    p, it, rz = z.copy(), 0, r @ z
    while np.linalg.norm(r) > 1e-12 * np.linalg.norm(b):
        q = J @ p
        a = rz / (p @ q)
        r -= a * q
        z = r / D
        rz, old = r @ z, rz
        p = z + rz / old * p
        it += 1
    return it


@pytest.mark.parametrize("n,sphere", [(5, False), (6, False), (9, False), (10, True), (14, False), (16, True)])
def test_residual(tmp_path, n, sphere):
    _, path = make_deck(tmp_path, n, sphere=(50.0, 50.0, 50.0, 20.0) if sphere else None)
    dk = mp.Deck.load(path)
    dense, sparse = context(dk), context(dk, mp.FE_SPARSE)
    rng = np.random.default_rng(n)
    for level in (0.0, 12.0):  # volts: the second's Boltzmann term is e^6 times the first's
        d, b = rng.normal(level, 0.05, dense.neq), rng.normal(size=dense.neq)
        y, st = solve(dense, d, b)
        J = dense_j(dense, d)
        assert holds(J, y, b)
        assert st.linear_iterations < by_diagonal(J, b) or level
        assert np.array_equal(y, solve(sparse, d, b)[0])
        assert np.array_equal(y, solve(dense, d, b)[0])


def test_thin_and_shuffled(tmp_path):
    kd, _ = make_deck(tmp_path, 9)
    rng = np.random.default_rng(3)
    p = rng.permutation(kd.n_nodes)
    pos = np.empty_like(kd.nodes_mm)
    pos[p] = kd.nodes_mm * (1e-3, 4e-4, 1e-4)
    fixed = p[np.concatenate([kd.wall_nodes, kd.sphere_nodes])]
    mesh = mp.Mesh.build(pos, p[kd.tets], p[kd.inlet_nodes], p[kd.inlet_tris], fixed)
    _, path = make_deck(tmp_path, 9)
    ctx = context(mp.Deck(mp.Deck.load(path).params, mesh, kd.sphere_nodes))
    d, b = rng.normal(0.0, 0.05, ctx.neq), rng.normal(size=ctx.neq)
    y, _ = solve(ctx, d, b)
    assert holds(dense_j(ctx, d), y, b)


def test_k_given_anew(tmp_path):
    """The solver's own copy of K follows a second setup of the context."""
    _, path = make_deck(tmp_path, 8)
    dk = mp.Deck.load(path)
    ctx = context(dk)
    K, F0 = ctx.fe_get("K"), ctx.fe_get("F0")
    rng = np.random.default_rng(1)
    d, b = rng.normal(0.0, 0.05, ctx.neq), rng.normal(size=ctx.neq)
    solve(ctx, d, b)
    ctx.fe_setup(**dk.fe_desc_arrays(None), K=3.0 * K, F0=F0)
    y, _ = solve(ctx, d, b)
    assert holds(dense_j(ctx, d), y, b)


def test_refused(tmp_path):
    """The iteration limit and an indefinite J are reported as by the plain iteration."""
    _, path = make_deck(tmp_path, 8)
    dk = mp.Deck.load(path)
    ctx = context(dk)
    K, F0 = ctx.fe_get("K"), ctx.fe_get("F0")
    d, b = np.zeros(ctx.neq), np.ones(ctx.neq)
    ctx.set_sparse_solver(1e-12, 4)
    with pytest.raises(mp.MpError) as e:
        solve(ctx, d, b)
    assert e.value.status == 5  # MP_ERR_NOT_CONVERGED
    ctx.set_sparse_solver()
    y, _ = solve(ctx, d, b)
    assert holds(dense_j(ctx, d), y, b)
    K[7, 7] = -K[7, 7]
    bad = context(dk, K=K, F0=F0)
    with pytest.raises(mp.MpError) as e:
        solve(bad, d, b)
    assert e.value.status == 6  # MP_ERR_SINGULAR
