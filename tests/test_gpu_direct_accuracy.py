"""GPU: the direct solve of an indefinite J whose elimination meets pivots far smaller
than its entries (a given K of the mesh's pattern): the sparse factorization does not
pivot, so its solution is refined, or the dense one taken, until it is as good as a
stable solve, in both forms and through both entry points.

Tolerance: a backward stable solve differs from numpy's by the condition number
(computed here, about 100) times 2^-53 times a modest factor for the 64 x 64 blocks'
sums, 1e2."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import make_deck
import minipic_b200 as mp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 12])
@pytest.mark.parametrize("small", [1e-3, 1e-5, 1e-7, 1e-10, 1e-13, 1e-16])
def test_small_pivots(tmp_path, n, small):
    _, path = make_deck(tmp_path, n)
    dk = mp.Deck.load(path)
    rng = np.random.default_rng(n)
    ctx = mp.Context(dk.mesh)
    ctx.fe_setup(**dk.fe_desc_arrays())
    d, b = rng.normal(0.0, 0.05, ctx.neq), rng.normal(size=ctx.neq)
    ctx.fe_set("d", d)
    ctx.build_j(mp.LAPACK)
    K, F0 = ctx.fe_get("K"), ctx.fe_get("F0")
    fp = np.diag(K - ctx.fe_get("J"))
    # a twelfth of the unknowns, no two of them neighbours, with next to no diagonal
    near, chosen = np.zeros(ctx.neq, bool), []
    for u in rng.permutation(ctx.neq):
        if not near[u] and len(chosen) < ctx.neq // 12:
            chosen.append(u)
            near[np.nonzero(K[u])[0]] = True
    K[chosen, chosen] = fp[chosen] + small * K[chosen, chosen]
    ctx.fe_setup(**dk.fe_desc_arrays(), K=K, F0=F0)
    ctx.fe_set("d", d)
    ctx.build_j(mp.LAPACK)
    J = ctx.fe_get("J")
    tol = 1e2 * 2.0 ** -53 * np.linalg.cond(J)
    ref = np.linalg.solve(J, b)
    scale = np.abs(ref).max()
    for form in (mp.FP64, mp.MIXED):
        ctx.build_j(mp.LAPACK)
        ctx.solve_linear(mp.LAPACK, form, b=b)
        assert np.abs(ctx.fe_get("y") - ref).max() <= tol * scale, form
    den = 1e10 * (1 + 0.1 * rng.standard_normal(dk.mesh.n_nodes))
    for form in (mp.FP64, mp.MIXED):
        ctx.fe_set("d", d)
        ctx.fe_set("F1", np.zeros(ctx.neq))
        ctx.compute_phi(mp.LAPACK, form, ion_den=den)
        ref = np.linalg.solve(J, ctx.fe_get("G"))
        assert np.abs(ctx.fe_get("y") - ref).max() <= tol * np.abs(ref).max(), form
