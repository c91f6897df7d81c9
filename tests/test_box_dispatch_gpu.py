"""Which merges k_box takes in a batch: by their poles (more than 512, and at
least 9/20 of the level's rows) and by the level's merges (levels of up to 1024
rows: from 8 merges of more than 768 rows on, 64 of more than 512).  Orders and
counts on both sides of each line; the repository's bar for eigenvalues."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


# Toeplitz keeps half the rows of its last merge: 512, 530, 768 and 770 poles;
# glued Wilkinson matrices keep less than 9/20 of theirs
@pytest.mark.parametrize("count", [7, 8, 63, 64])
@pytest.mark.parametrize("kind,orders", [("toeplitz", (1024, 1060, 1536, 1541)), ("disorder", (600, 790, 1000, 1024)),
                                         ("glued", (1155, 1260, 1491, 2037))])
def test_batch(solver, count, kind, orders):
    import torch

    rng = np.random.default_rng(count)
    sizes = [orders[i % len(orders)] for i in range(count)]
    off = np.concatenate([[0], np.cumsum(sizes)])
    D = np.full(off[-1], 2.0) if kind == "toeplitz" else 0.05 * rng.standard_normal(off[-1])
    E = np.ones(off[-1])
    if kind == "glued":  # W21 after W21: every order is a multiple of 21
        D = np.tile(np.abs(np.arange(21) - 10.0), off[-1] // 21)
        E[20::21] = 1e-8
    E[off[1:] - 1] = 0.0
    Dt, Et = torch.tensor(D, device="cuda"), torch.tensor(E, device="cuda")
    W = solver.dstebr_batched(off, Dt, Et).clone()
    for b in range(len(orders)):
        lo, hi = off[b], off[b + 1]
        ref = np.sort(oracle.dsterf(D[lo:hi], E[lo:hi - 1]))
        assert np.abs(W[lo:hi].cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
    if kind != "disorder":  # equal matrices have equal spectra wherever they lie
        for b in range(len(orders), count):
            first = off[b % len(orders)]
            assert torch.equal(W[off[b]:off[b + 1]], W[first:first + sizes[b]])
    ws = solver.batched_workspace(off, checkpoints=True)
    assert torch.equal(solver.dstebr_batched(off, Dt, Et, workspace=ws), W)
