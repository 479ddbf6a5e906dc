"""GPU: the direct solve J y = G by the sparse factorization (nested dissection,
64 x 64 tiles), against numpy's dense solve of the downloaded J, at sizes from
one partly filled tile to a few elimination levels; in meshes whose numbering
or missing node positions leave the dissection little to go by; and the calls
that the dense factorization still takes.

Tolerance: both solves are backward stable on J with condition below 1e3 here
(numpy's condition number is checked), so the relative difference is below
1e3 * 2^-53 * a growth of 1e2 = 1e-11."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import make_deck
import minipic_b200 as mp

pytestmark = pytest.mark.gpu
TOL = 1e-11


def context(dk, sphere=False, **kw):
    ctx = mp.Context(dk.mesh)
    ctx.fe_setup(**dk.fe_desc_arrays(-10.0 if sphere else None), **kw)
    return ctx


def state(ctx, seed):
    rng = np.random.default_rng(seed)
    ctx.fe_set("d", rng.normal(0.0, 0.05, ctx.neq))
    return rng.normal(size=ctx.neq)


def rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


def check(ctx, seed):
    b = state(ctx, seed)
    for form in (mp.FP64, mp.MIXED):
        ctx.build_j(mp.LAPACK)
        J = ctx.fe_get("J")
        assert np.linalg.cond(J) < 1e3
        ref = np.linalg.solve(J, b)
        st = ctx.solve_linear(mp.LAPACK, form, b=b)
        assert rel(ctx.fe_get("y"), ref) < TOL, (form, rel(ctx.fe_get("y"), ref))
        assert st.linear_residual * ctx.neq <= 1e-12 * np.linalg.norm(b)
    return J


@pytest.mark.parametrize("n,sphere", [(2, False), (3, False), (4, False), (5, False), (8, False), (9, False),
                                      (10, True), (12, False)])
def test_against_numpy(tmp_path, n, sphere):
    kd, path = make_deck(tmp_path, n, sphere=(50.0, 50.0, 50.0, 20.0) if sphere else None)
    check(context(mp.Deck.load(path), sphere), n)


class NoPositions(mp.Mesh):
    def desc(self):
        d = super().desc()
        d.node_pos, d.node_pos_stride = None, 0
        return d


@pytest.mark.parametrize("positions", [True, False])
def test_shuffled_numbering(tmp_path, positions):
    """Nodes numbered at random (the dissection cannot rely on the order), with
    positions and without (levels of a breadth-first search instead)."""
    kd, path = make_deck(tmp_path, 9)
    rng = np.random.default_rng(3)
    p = rng.permutation(kd.n_nodes)
    pos = np.empty_like(kd.nodes_mm)
    pos[p] = kd.nodes_mm / 1000.0
    fixed = p[np.concatenate([kd.wall_nodes, kd.sphere_nodes])]
    mesh = mp.Mesh.build(pos, p[kd.tets], p[kd.inlet_nodes], p[kd.inlet_tris], fixed)
    if not positions:
        mesh.__class__ = NoPositions
    check(context(mp.Deck(mp.Deck.load(path).params, mesh, kd.sphere_nodes)), 4)


def test_given_k(tmp_path):
    """K from the caller: the mesh's own takes the sparse factorization; one with a
    coupling between two unknowns of no common tet, or an unsymmetric one (its
    lower triangle counts), the dense one."""
    kd, path = make_deck(tmp_path, 8)
    dk = mp.Deck.load(path)
    ref = context(dk)
    K, F0 = ref.fe_get("K"), ref.fe_get("F0")
    J = check(context(dk, K=K, F0=F0), 5)
    far = np.argwhere(J[-1] == 0)[0, 0]
    K2 = K.copy()
    K2[-1, far] = K2[far, -1] = 0.1 * K[0, 0]
    K3 = K.copy()
    i, j = np.argwhere(np.triu(K, 1))[7]
    K3[i, j] *= 2.0
    for Kx in (K2, K3):
        ctx = context(dk, K=Kx, F0=F0)
        b = state(ctx, 6)
        ctx.build_j(mp.LAPACK)
        Jx = np.tril(ctx.fe_get("J"))
        Jx += np.tril(Jx, -1).T
        ctx.solve_linear(mp.LAPACK, mp.FP64, b=b)
        assert rel(ctx.fe_get("y"), np.linalg.solve(Jx, b)) < TOL


def test_singular_is_still_reported(tmp_path):
    """A row of zeros in K whose Boltzmann term underflows: no factorization has a pivot for it."""
    kd, path = make_deck(tmp_path, 5)
    dk = mp.Deck.load(path)
    ref = context(dk)
    K, F0 = ref.fe_get("K"), ref.fe_get("F0")
    K[7, :] = K[:, 7] = 0.0
    ctx = context(dk, K=K, F0=F0)
    d = np.zeros(ctx.neq)
    d[7] = -1e5  # exp(d / kTe) = 0
    ctx.fe_set("d", d)
    ctx.build_j(mp.LAPACK)
    with pytest.raises(mp.MpError) as e:
        ctx.solve_linear(mp.LAPACK, mp.FP64, b=np.ones(ctx.neq))
    assert e.value.status == 6  # MP_ERR_SINGULAR


def test_j_of_a_step(tmp_path):
    """computePhi forms no dense J, but the J of the step can be downloaded, and a
    Gauss-Seidel step's J solved with, as when it was formed; a J is used up by
    one direct FP64 solve."""
    kd, path = make_deck(tmp_path, 6)
    ctx = context(mp.Deck.load(path))
    den = np.full(ctx.mesh.n_nodes, 1e10)
    K = ctx.fe_get("K")
    off = ~np.eye(ctx.neq, dtype=bool)
    ctx.compute_phi(mp.LAPACK, mp.FP64, ion_den=den)
    J = ctx.fe_get("J")
    assert np.array_equal(J[off], K[off]) and np.all(J[~off] != K[~off])
    with pytest.raises(mp.MpError) as e:
        ctx.solve_linear(mp.LAPACK, mp.FP64)
    assert e.value.status == 7
    ctx.compute_phi(mp.GAUSS_SEIDEL, mp.FP64, ion_den=den)
    J = ctx.fe_get("J")
    ctx.compute_phi(mp.LAPACK, mp.MIXED, ion_den=den)  # its own Boltzmann term
    b = np.random.default_rng(1).normal(size=ctx.neq)
    ctx.solve_linear(mp.LAPACK, mp.FP64, b=b)
    assert rel(ctx.fe_get("y"), np.linalg.solve(J, b)) < TOL


@pytest.mark.parametrize("n,sphere", [(2, False), (5, False), (8, False), (10, True)])
@pytest.mark.parametrize("method", [mp.LAPACK, mp.GAUSS_SEIDEL, mp.SPARSE_CG])
def test_step_terms_bitwise(tmp_path, n, sphere, method):
    """The fused step's F1 and G are those of the separate entry points bit for bit,
    and its update is d - y and g + d in one rounding each."""
    kd, path = make_deck(tmp_path, n, sphere=(50.0, 50.0, 50.0, 20.0) if sphere else None)
    dk = mp.Deck.load(path)
    ctx = context(dk, sphere)
    rng = np.random.default_rng(n)
    den = 1e10 * (1 + 0.1 * rng.standard_normal(dk.mesh.n_nodes))
    d, F1 = rng.normal(0.0, 0.5, ctx.neq), rng.normal(0.0, 1e-3, ctx.neq)
    ctx.fe_set("d", d)
    ctx.fe_set("F1", F1)
    ctx.build_f1(den)
    ctx.residual()
    ref = ctx.fe_get("F1"), ctx.fe_get("G")
    ctx.fe_set("F1", F1)
    ctx.compute_phi(method, mp.FP64, ion_den=den)
    assert np.array_equal(ctx.fe_get("F1"), ref[0]) and np.array_equal(ctx.fe_get("G"), ref[1])
    ID = dk.mesh.fe_geometry()[0]
    y, now, uh, g = (ctx.fe_get(k) for k in ("y", "d", "uh", "g"))
    assert np.array_equal(now, d - y)
    assert np.array_equal(uh, np.where(ID >= 0, g + now[ID], g))


def test_refinement(tmp_path):
    """Right-hand sides whose solution is far larger (inverse iteration, J's smoothest
    modes): the mixed form refines, by forward and backward solves with the factor."""
    kd, path = make_deck(tmp_path, 16)
    ctx = context(mp.Deck.load(path))
    b = state(ctx, 7)
    ctx.build_j(mp.LAPACK)
    J = ctx.fe_get("J")
    most = 0
    for _ in range(8):
        ctx.build_j(mp.LAPACK)
        st = ctx.solve_linear(mp.LAPACK, mp.MIXED, b=b)
        y = ctx.fe_get("y")
        assert np.linalg.norm(b - J @ y) <= 1e-13 * np.linalg.norm(b)
        most = max(most, st.linear_iterations)
        last, b = b, y / np.linalg.norm(y)
    assert most > 1
    assert rel(y, np.linalg.solve(J, last)) < TOL
