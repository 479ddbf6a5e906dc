"""GPU: the solvers that take a call where the sparse ones do not, at sizes of many
blocks: the dense LDL^T in FP64 past one 1,024-column super-panel (a K with one
coupling outside the mesh's pattern) and in the mixed form's explicit arithmetics,
the dense Gauss-Seidel sweeps (such a K, more rows than a cluster holds, rows with
more than 14 neighbours), conjugate gradients by J's diagonal (a mesh without node
positions, a thin one between fixed planes).  And the sparse solvers on a mesh that is no lattice (Delaunay).  The
number of launches tells which solver ran.

Tolerances: a direct solve is backward stable (the mixed form refined to 1e-14) on J
with condition below 1e3 (computed for the Delaunay mesh: 123 and 876): 1e-11 relative of
the largest value; Gauss-Seidel and conjugate gradients as in their own tests."""
from __future__ import annotations

import numpy as np
import pytest
import torch
from scipy.spatial import Delaunay

from conftest import make_deck
from test_gpu_gauss_seidel import run
from test_gpu_multilevel_cg import by_diagonal, holds
from test_gpu_sparse_direct import NoPositions
import minipic_b200 as mp

pytestmark = pytest.mark.gpu
TOL = 1e-11


def context(dk, **kw):
    ctx = mp.Context(dk.mesh)
    ctx.fe_setup(**dk.fe_desc_arrays(), **kw)
    ctx.fe_set("d", np.random.default_rng(2).normal(0.0, 0.05, ctx.neq))
    return ctx


def far_coupling(dk, share):
    """A context whose K couples the last unknown to one that it shares no tet with."""
    ref = context(dk)
    K, F0 = ref.fe_get("K"), ref.fe_get("F0")
    ref.close()
    far = np.argwhere(K[-1] == 0)[0, 0]
    K[-1, far] = K[far, -1] = share * K[0, 0]
    return context(dk, K=K, F0=F0)


def launches(ctx, method, form=mp.FP64, b=None):
    ctx.build_j(method)
    before = ctx.launches()
    try:
        ctx.solve_linear(method, form, b=b)
    except mp.MpError as e:
        assert e.status == 5  # the sweep limit
    return ctx.launches() - before


def unstructured(tmp_path, m):
    """Delaunay mesh of a box's m^3 points, the inner ones moved at random."""
    rng = np.random.default_rng(0)
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3).astype(float)
    inner = (g > 0) & (g < m - 1)
    p = (g + np.where(inner, rng.uniform(-0.3, 0.3, g.shape), 0.0)) * (0.1 / (m - 1))
    t = Delaunay(p).simplices
    e = p[t[:, 1:]] - p[t[:, :1]]
    t = t[np.abs(np.linalg.det(e)) > 1e-5 * (0.1 / (m - 1)) ** 3]
    faces, count = np.unique(np.sort(np.concatenate([t[:, [0, 1, 2]], t[:, [0, 1, 3]], t[:, [0, 2, 3]], t[:, [1, 2, 3]]]), 1),
                             axis=0, return_counts=True)
    faces = faces[count == 1]
    mesh = mp.Mesh.build(p, t, np.nonzero(p[:, 0] == 0)[0], faces[(p[faces][:, :, 0] == 0).all(1)],
                         np.nonzero(p[:, 0] == p[:, 0].max())[0])
    _, path = make_deck(tmp_path, 2)
    return mp.Deck(mp.Deck.load(path).params, mesh, np.zeros(0, dtype=np.int64))


@pytest.mark.parametrize("n", [12, 20], ids=["1859", "8379"])
def test_dense_fp64(tmp_path, n):
    _, path = make_deck(tmp_path, n)
    ctx = far_coupling(mp.Deck.load(path), 0.1)
    b = np.random.default_rng(n).normal(size=ctx.neq)
    ctx.build_j(mp.LAPACK)
    J = torch.as_tensor(ctx.fe_get("J"), device="cuda")
    ref = torch.linalg.solve(J, torch.as_tensor(b, device="cuda")).cpu().numpy()
    assert launches(ctx, mp.LAPACK, b=b) > ctx.neq // 64
    assert np.abs(ctx.fe_get("y") - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("n", [12, 20], ids=["1859", "8379"])
@pytest.mark.parametrize("factor", [mp.MIXED_TF32, mp.MIXED_FP16, mp.MIXED_TF32X3], ids=["tf32", "fp16", "tf32x3"])
def test_dense_mixed(tmp_path, n, factor):
    _, path = make_deck(tmp_path, n)
    ctx = context(mp.Deck.load(path))
    b = np.random.default_rng(n).normal(size=ctx.neq)
    ctx.build_j(mp.LAPACK)
    J = torch.as_tensor(ctx.fe_get("J"), device="cuda")
    ref = torch.linalg.solve(J, torch.as_tensor(b, device="cuda")).cpu().numpy()
    ctx.set_mixed_factor(factor)
    assert launches(ctx, mp.LAPACK, mp.MIXED, b) > ctx.neq // 64
    assert np.abs(ctx.fe_get("y") - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("case", ["far_1859", "rows_8379", "wide_1089"])
def test_dense_sweeps(tmp_path, case):
    if case == "far_1859":
        _, path = make_deck(tmp_path, 12)
        ctx, limit = far_coupling(mp.Deck.load(path), 0.01), 27
    elif case == "rows_8379":
        _, path = make_deck(tmp_path, 20)
        ctx, limit = context(mp.Deck.load(path)), 2
    else:
        ctx, limit = context(unstructured(tmp_path, 11)), 27
    assert str(ctx.neq) in case
    b = np.random.default_rng(1).normal(size=ctx.neq) * 0.1
    run(ctx, b, limit)
    assert launches(ctx, mp.GAUSS_SEIDEL, b=b) > 3  # one in the cluster form


@pytest.mark.parametrize("n,mesh", [(9, "no positions"), (14, "no positions"), (6, "thin"), (12, "thin")])
def test_conjugate_gradients_by_the_diagonal(tmp_path, n, mesh):
    kd, path = make_deck(tmp_path, n)
    dk = mp.Deck.load(path)
    if mesh == "thin":
        dk = mp.Deck(dk.params, mp.Mesh.build(kd.nodes_mm * (5e-5, 1e-3, 1e-3), kd.tets, kd.inlet_nodes, kd.inlet_tris,
                                              kd.wall_nodes), kd.sphere_nodes)
    else:
        dk.mesh.__class__ = NoPositions
    ctx = context(dk)
    b = np.random.default_rng(n).normal(size=ctx.neq)
    ctx.build_j(mp.LAPACK)
    J = ctx.fe_get("J")
    ctx.build_j(mp.SPARSE_CG)
    st = ctx.solve_linear(mp.SPARSE_CG, mp.FP64, b=b)
    assert holds(J, ctx.fe_get("y"), b)
    expected = by_diagonal(J, b)  # the levels take less than 2/3 of them, or in the thin boxes more
    assert abs(st.linear_iterations - expected) <= 0.05 * expected + 2


@pytest.mark.parametrize("m", [6, 11])
def test_sparse_solvers_off_the_lattice(tmp_path, m):
    ctx = context(unstructured(tmp_path, m))
    rows = np.diff(ctx.fe_sparse_matrix()[0])
    assert rows.max() > 18 and rows.min() < 12
    b = np.random.default_rng(m).normal(size=ctx.neq)
    ctx.build_j(mp.LAPACK)
    J = ctx.fe_get("J")
    assert np.linalg.cond(J) < 1e3
    ref = np.linalg.solve(J, b)
    for form in (mp.FP64, mp.MIXED):
        assert launches(ctx, mp.LAPACK, form, b) < 10
        assert np.abs(ctx.fe_get("y") - ref).max() <= TOL * np.abs(ref).max()
    ctx.build_j(mp.SPARSE_CG)
    ctx.solve_linear(mp.SPARSE_CG, mp.FP64, b=b)
    assert holds(J, ctx.fe_get("y"), b)
