"""GPU: solves on a device with almost no memory left.  A direct solve whose sparse
factor does not fit is taken over by the dense one where that has its memory, is
refused with an error where not, and runs as ever once there is room again.

Tolerance: the dense and the sparse solve are backward stable on J with condition
below 1e3 (the 20^3 Kuhn box), so y differs by less than 1e3 * 2^-53 * a growth of
1e2 = 1e-11 of its largest value."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import make_deck
import minipic_b200 as mp

pytestmark = pytest.mark.gpu


def fill(left):
    """Holds the device's memory but for about `left` bytes."""
    held, size = [], 1 << 35
    while size >= 1 << 21:
        free = torch.cuda.mem_get_info()[0]
        if free < left + size:
            size >>= 1
            continue
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size >>= 1
    return held


def context(dk):
    ctx = mp.Context(dk.mesh)
    ctx.fe_setup(**dk.fe_desc_arrays())
    return ctx


def step(ctx, method=mp.LAPACK, form=mp.FP64):
    rng = np.random.default_rng(3)
    den = 1e10 * (1 + 0.1 * rng.standard_normal(ctx.mesh.n_nodes))
    ctx.fe_set("d", rng.normal(0.0, 0.05, ctx.neq))
    ctx.fe_set("F1", np.zeros(ctx.neq))
    before = ctx.launches()
    ctx.compute_phi(method, form, ion_den=den)
    return ctx.fe_get("y"), ctx.launches() - before


def test_direct_solve(tmp_path):
    _, path = make_deck(tmp_path, 20)
    dk = mp.Deck.load(path)
    first = context(dk)
    ref, few = step(first)
    first.close()
    ctx, dense = context(dk), context(dk)
    # the dense factorization's memory, without the sparse factor's
    dense.set_mixed_factor(mp.MIXED_TF32)
    step(dense, form=mp.MIXED)
    dense.set_mixed_factor(mp.MIXED_AUTO)
    dense.build_j(mp.LAPACK)
    held = fill(24 << 20)
    try:
        for _ in range(2):
            with pytest.raises(mp.MpError):
                step(ctx)
        y, many = step(dense)
    finally:
        del held
        torch.cuda.empty_cache()
    assert many > 10 * few
    assert np.abs(y - ref).max() <= 1e-11 * np.abs(ref).max()
    for c in (ctx, dense):
        y, count = step(c)
        assert count == few
        assert np.array_equal(y, ref)
