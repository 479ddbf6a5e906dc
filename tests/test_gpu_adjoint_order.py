"""GPU: the adjoint's results do not depend on the order particles are given in
(slots are laid out by cell inside), for batch sizes around a warp, a block and
a CTA's run, entering at different steps, with a checkpoint interval that does
not divide the steps.

Tolerance: the same terms in another order of the FP64 atomics: 1e-12 relative
of the largest value."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import make_deck
import minipic_b200 as mp
from minipic_b200 import adjoint, kuhn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1,), (31, 33, 2), (256, 257, 1), (5000, 300, 700, 13)])
def test_order_does_not_matter(tmp_path, sizes):
    kd, path = make_deck(tmp_path, 6)
    dk = mp.Deck.load(path)
    rng = np.random.default_rng(sum(sizes))
    batches = []
    for k, n in enumerate(sizes):
        pos = rng.uniform(1e-4, 0.0999, size=(n, 3))
        vel = rng.normal(0.0, 2e4, size=(n, 3)) + [7e4, 0, 0]
        batches.append((2 * k, k % 2 == 1, pos, vel, kuhn.locate(kd, pos).astype(np.int32)))
    _, nx, _, _ = dk.mesh.fe_geometry()
    phi = -50.0 * dk.mesh.node_pos[:, 0] + rng.normal(0.0, 0.1, dk.mesh.n_nodes)
    bar = rng.normal(size=dk.mesh.n_nodes)
    out = []
    for order in ("given", "reversed", "by cell"):
        ctx = mp.Context(dk.mesh)
        adj = adjoint.Adjoint(ctx, 8, 3, mp.QE / (16 * mp.AMU), 16 * mp.AMU, 1e-7, 10.0, [1.0, 0, 0],
                              adjoint.wall_nodes_of(dk.mesh), nx=nx)
        for first, inj, pos, vel, cell in batches:
            o = {"given": np.arange(len(cell)), "reversed": np.arange(len(cell))[::-1], "by cell": np.argsort(cell)}[order]
            adj.add_particles(first, inj, pos[o], vel[o], cell[o])
        den, st = adj.forward(phi, 7000.0)
        pb, vb = adj.backward(bar, 1e6)
        dd, df = adj.tangent(bar, 3.0)
        assert st.slots == sum(sizes) and st.alive + st.wall_exits + st.other_exits == st.slots
        out.append((den, pb, dd, np.array([st.flux, vb, df]), (st.alive, st.wall_exits, st.other_exits)))
    for other in out[1:]:
        assert other[4] == out[0][4]
        for a, b in zip(out[0][:3], other[:3]):
            assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max()
        assert np.all(np.abs(out[0][3] - other[3]) <= 1e-12 * np.abs(out[0][3]))
