"""GPU: adjoint particles come into their slots in pieces: several pieces with an odd
rest give the same as many calls, the staging takes little device memory, and
particles in device memory are read after the work on them in the default stream,
also where the cells are on the host.

Tolerance: the same terms in another order of the FP64 atomics: 1e-12 relative
of the largest value."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import make_deck
import minipic_b200 as mp
from minipic_b200 import adjoint, kuhn

pytestmark = pytest.mark.gpu

PIECE = 1 << 19
STEPS = 2
SLOT_BYTES = 6 * 8 + 2 * 4 + 1 + 2 * 4 + 1  # inputs and outcomes; no checkpoint in two steps


@pytest.fixture(scope="module")
def case(tmp_path_factory):
    kd, path = make_deck(tmp_path_factory.mktemp("adj"), 6)
    dk = mp.Deck.load(path)
    n = 6 * PIECE + 7
    rng = np.random.default_rng(1)
    pos = rng.uniform(1e-4, 0.0999, size=(n, 3))
    vel = rng.normal(0.0, 2e4, size=(n, 3)) + [7e4, 0, 0]
    return dk, pos, vel, kuhn.locate(kd, pos).astype(np.int32)


def new(dk):
    ctx = mp.Context(dk.mesh)
    _, nx, _, _ = dk.mesh.fe_geometry()
    return ctx, adjoint.Adjoint(ctx, STEPS, STEPS, mp.QE / (16 * mp.AMU), 16 * mp.AMU, 1e-7, 10.0, [1.0, 0, 0],
                                adjoint.wall_nodes_of(dk.mesh), nx=nx)


def results(dk, adj):
    rng = np.random.default_rng(2)
    den, st = adj.forward(-50.0 * dk.mesh.node_pos[:, 0] + rng.normal(0.0, 0.1, dk.mesh.n_nodes), 7000.0)
    phi_bar, _ = adj.backward(rng.normal(size=dk.mesh.n_nodes), 1e6)
    return den, phi_bar, (st.slots, st.alive, st.wall_exits, st.other_exits)


def same(a, b):
    assert a[2] == b[2]
    for u, v in zip(a[:2], b[:2]):
        assert np.abs(u - v).max() <= 1e-12 * np.abs(v).max()


def test_pieces(case):
    dk, pos, vel, cell = case
    ctx, adj = new(dk)
    free = torch.cuda.mem_get_info()[0]
    adj.add_particles(0, False, pos, vel, cell)
    # and the allocator's rounding
    assert free - torch.cuda.mem_get_info()[0] <= SLOT_BYTES * len(cell) + (64 << 20)
    one = results(dk, adj)
    ctx.close()
    ctx, adj = new(dk)
    for part in np.array_split(np.arange(len(cell)), 17):
        adj.add_particles(0, False, pos[part], vel[part], cell[part])
    same(one, results(dk, adj))


def test_after_the_default_streams_work(case):
    dk, pos, vel, cell = (a[:100_001] if isinstance(a, np.ndarray) else a for a in case)
    ctx, adj = new(dk)
    adj.add_particles(0, False, pos, vel, cell)
    ref = results(dk, adj)
    ctx.close()
    ctx, adj = new(dk)
    p, v = torch.full(pos.shape, 0.05, dtype=torch.float64, device="cuda"), torch.zeros(pos.shape, dtype=torch.float64, device="cuda")
    p_in, v_in = torch.as_tensor(pos, device="cuda"), torch.as_tensor(vel, device="cuda")
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)  # about 50 ms
    p.copy_(p_in)
    v.copy_(v_in)
    ctx._c(mp.lib().mp_adjoint_add_particles(ctx.h, 0, 0, cell.size, p.data_ptr(), v.data_ptr(), mp._p(cell)))
    same(results(dk, adj), ref)
