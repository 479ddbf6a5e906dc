"""GPU: Gauss-Seidel on a mesh numbered in other orders than by coordinate: the cluster
kernel where its levels are few enough to be the faster way (also with rows that
keep their value), the dense sweeps where not, and the row-by-row iterates in both.
The number of launches tells which ran."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import make_deck
from test_gpu_gauss_seidel import run
import minipic_b200 as mp

pytestmark = pytest.mark.gpu


def context(tmp_path, n, order, kept=()):
    kd, path = make_deck(tmp_path, n)
    rng = np.random.default_rng(3)
    g = np.arange(kd.n_nodes)
    if order == "random":
        p = rng.permutation(kd.n_nodes)
    elif order == "slabs":  # at random within each plane of the last axis
        p = np.empty_like(g)
        p[np.argsort(g // (n + 1) ** 2 + 0.999 * rng.random(kd.n_nodes), kind="stable")] = g
    else:  # the last axis fastest
        m = n + 1
        p = g // m ** 2 + m * (g // m % m + m * (g % m))
    pos = np.empty_like(kd.nodes_mm)
    pos[p] = kd.nodes_mm / 1000.0
    mesh = mp.Mesh.build(pos, p[kd.tets], p[kd.inlet_nodes], p[kd.inlet_tris], p[kd.wall_nodes])
    dk = mp.Deck(mp.Deck.load(path).params, mesh, kd.sphere_nodes)
    ctx = mp.Context(dk.mesh)
    ctx.fe_setup(**dk.fe_desc_arrays())
    d = rng.normal(0.0, 0.05, ctx.neq)
    ctx.fe_set("d", d)
    if kept:
        ctx.build_j(mp.GAUSS_SEIDEL)
        K, F0 = ctx.fe_get("K"), ctx.fe_get("F0")
        fp = np.diag(K - ctx.fe_get("J"))
        for u in kept:
            K[u, u] = fp[u]
        ctx.fe_setup(**dk.fe_desc_arrays(), K=K, F0=F0)
        ctx.fe_set("d", d)
    return ctx


@pytest.mark.parametrize("n,order,kept,limit,cluster", [
    (5, "random", (), 27, True), (8, "random", (), 27, False), (8, "slabs", (), 27, False),
    (3, "random", (), 27, True), (8, "last axis fastest", (), 27, True), (8, "last axis fastest", (0, 11, 566), 3, True),
    (12, "random", (), 27, True), (12, "slabs", (1858,), 3, True)])
def test_orders(tmp_path, n, order, kept, limit, cluster):
    ctx = context(tmp_path, n, order, kept)
    b = np.random.default_rng(n).normal(size=ctx.neq) * 0.1
    run(ctx, b, limit)
    ctx.build_j(mp.GAUSS_SEIDEL)
    before = ctx.launches()
    try:
        ctx.solve_linear(mp.GAUSS_SEIDEL, mp.FP64, b=b)
    except mp.MpError as e:
        assert e.status == 5  # the sweep limit
    assert (ctx.launches() - before == 1) == cluster
