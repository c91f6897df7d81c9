"""k_box where a box's interval straddles clusters of poles (listed boxes,
csrc/brdc_box.cuh: more near poles than six boxes'): their roots run with more
lanes.  Poles in two clusters (one straddling box), in up to 16 (many of them),
and merges so small that most boxes have no far part."""
import math

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _matrix(kind, n):
    if kind == "two":  # dimers, weakly coupled: eigenvalues near +-sqrt(2)
        return np.tile([1.0, -1.0], n // 2 + 1)[:n], np.tile([1.0, 1e-9], n // 2 + 1)[:n - 1]
    rng = np.random.default_rng(7)
    if kind == "sixteen":  # a 16-row block repeated
        return np.tile(rng.standard_normal(16), n // 16 + 1)[:n], np.tile(rng.standard_normal(16), n // 16 + 1)[:n - 1]
    d, e = np.tile(np.abs(np.arange(21) - 10.0), n // 21 + 1)[:n], np.ones(n - 1)
    e[20::21] = 1e-8  # Wilkinson's W21, glued
    return d, e


@pytest.mark.parametrize("kind", ["two", "sixteen", "glued"])
@pytest.mark.parametrize("n", [1100, 3000, 9001, 20000])
def test_against_lapack_and_direct_sums(solver, kind, n):
    """1e-12 of the norm against LAPACK; against the per-level kernels, which
    sum every pole directly, 16 eps of the norm a level (the bound of
    test_box_gpu.py).  A checkpointing solve is the plain one bit for bit."""
    import torch

    d, e = _matrix(kind, n)
    D, E = torch.tensor(d, device="cuda"), torch.tensor(e, device="cuda")
    W = solver.dstebr(D, E).clone()
    assert solver.info(n) == 0
    norm = float(W.abs().max())
    if n <= 9001:
        ref = np.sort(oracle.dsterf(d, e))
        assert np.abs(W.cpu().numpy() - ref).max() <= 1e-12 * norm
    assert torch.equal(solver.dstebr(D, E, workspace=solver.new_checkpoint_workspace(n)), W)
    tuning = solver.tuning()
    try:
        solver.set_tuning(fused_level_rows=0)
        V = solver.dstebr(D, E)
    finally:
        solver.set_tuning(**tuning)
    levels = math.ceil(math.log2(n / 16))
    assert float((W - V).abs().max()) <= levels * 16 * np.finfo(float).eps * norm


@pytest.mark.parametrize("kind", ["two", "sixteen"])
def test_batch(solver, kind):
    """Merges of different matrices in one level, each with listed boxes."""
    import torch

    orders = [3000, 1025, 2111, 4097]
    off = np.concatenate([[0], np.cumsum(orders)])
    D, E = np.empty(off[-1]), np.zeros(off[-1])
    for b, n in enumerate(orders):
        D[off[b]:off[b + 1]], E[off[b]:off[b + 1] - 1] = _matrix(kind, n)
    W = solver.dstebr_batched(off, torch.tensor(D, device="cuda"), torch.tensor(E, device="cuda")).cpu().numpy()
    for b in range(len(orders)):
        lo, hi = off[b], off[b + 1]
        ref = np.sort(oracle.dsterf(D[lo:hi], E[lo:hi - 1]))
        assert np.abs(W[lo:hi] - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("kind", ["two", "sixteen"])
def test_vectors(solver, kind):
    """Loewner weights and rows of inner merges: the bars of the eigenvector
    tests (orthogonality 1e-11, residual 1e-12 of the norm)."""
    import torch

    d, e = _matrix(kind, 5000)
    D, E = torch.tensor(d, device="cuda"), torch.tensor(e, device="cuda")
    W, Z = solver.dstebr_vectors(D, E)
    TZ = D[:, None] * Z
    TZ[:-1] += E[:, None] * Z[1:]
    TZ[1:] += E[:, None] * Z[:-1]
    assert float((TZ - Z * W).abs().max()) < 1e-12 * float(W.abs().max())
    gram = Z.T @ Z
    gram.diagonal().sub_(1.0)
    assert float(gram.abs().max()) < 1e-11
