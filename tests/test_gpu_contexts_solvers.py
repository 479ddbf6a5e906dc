"""GPU: two contexts on meshes of different sizes, driven at the same time from two
host threads, solve by each of the sparse methods as each does alone: launch
settings belong to a kernel in the process, so one context's may not be another's
limit.  Many short calls, so that the threads' launches meet in every order.

The solvers' sums have a fixed order: bit for bit."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from conftest import make_deck
import minipic_b200 as mp

pytestmark = pytest.mark.gpu

CALLS = 150


def _run(dk, method, out):
    ctx = mp.Context(dk.mesh)
    ctx.fe_setup(**dk.fe_desc_arrays())
    rng = np.random.default_rng(dk.mesh.n_nodes)
    den = 1e10 * (1 + 0.1 * rng.standard_normal(dk.mesh.n_nodes))
    d, zero = rng.normal(0.0, 0.05, ctx.neq), np.zeros(ctx.neq)
    res = []
    try:
        for _ in range(CALLS):
            ctx.fe_set("d", d)
            ctx.fe_set("F1", zero)
            ctx.compute_phi(method, mp.FP64, ion_den=den)
            res.append(ctx.fe_get("d"))
    except mp.MpError as e:
        res.append(e)
    ctx.close()
    out.append(res)


@pytest.mark.parametrize("method", [mp.SPARSE_CG, mp.GAUSS_SEIDEL, mp.LAPACK],
                         ids=["sparse_cg", "gauss_seidel", "lapack"])
def test_two_sizes_on_two_threads(tmp_path, method):
    decks = []
    for n in (6, 10):
        _, path = make_deck(tmp_path / str(n), n)
        decks.append(mp.Deck.load(path))
    alone = []
    for dk in decks:
        _run(dk, method, alone)
    outs = [[], []]
    threads = [threading.Thread(target=_run, args=(dk, method, out)) for dk, out in zip(decks, outs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for out, one in zip(outs, alone):
        assert len(out) == 1, "a thread failed"
        for x in [*out[0], *one]:
            assert not isinstance(x, Exception), x
        assert len(out[0]) == CALLS
        for x in [*out[0], *one]:
            assert np.array_equal(x, one[0])
