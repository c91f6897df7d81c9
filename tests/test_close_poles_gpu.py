"""Merges above 2048 rows that rotate close poles out of a short active list
(k_level's level_load_active and level_poles): every CTA of the cluster takes
its own copy of the list, and in a checkpointing solve CTA 0 writes the
rotated one back.

A random matrix that is its own mirror image (d and |e| symmetric about the
middle) gives its top merge two equal child spectra, of which a few dozen
poles in close pairs survive the small-z test; one made of equal mirrored
blocks does so at every level above a block."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
REPEATS = 20


def _mirrored(n, rng):
    d, e = rng.standard_normal(n), rng.standard_normal(n - 1)
    d[n - n // 2:] = d[:n // 2][::-1]
    e[n - 1 - (n - 1) // 2:] = e[:(n - 1) // 2][::-1]
    return d, e


def _matrix(n, block):
    rng = np.random.default_rng(n)
    if block == n:
        return _mirrored(n, rng)
    d, e = _mirrored(block, rng)
    return np.tile(d, n // block), np.tile(np.append(e, 0.7), n // block)[:-1]


CASES = [(4096, 4096), (6001, 6001), (9000, 9000), (10000, 2500), (20000, 20000)]


@pytest.mark.parametrize("n,block", CASES)
def test_checkpointing_solve_is_the_plain_one(solver, n, block):
    import torch

    d, e = _matrix(n, block)
    D, E = torch.tensor(d, device="cuda"), torch.tensor(e, device="cuda")
    plain = solver.dstebr(D, E).clone()
    ref = np.sort(oracle.dsterf(d, e))
    assert np.abs(plain.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
    ws = solver.new_checkpoint_workspace(n)
    for _ in range(REPEATS):
        assert torch.equal(solver.dstebr(D, E, workspace=ws), plain)
    # the case is what it is meant to be: rotations out of short lists
    rotated = 0
    for lv in solver.diagnostics(n, ws)["level"]:
        if lv["size_sum"] > 2048 * lv["merge_count"]:
            assert lv["dd_before_sum"] <= 1024 * lv["merge_count"]
            rotated += lv["close_deflated_total"]
    assert rotated > 0


@pytest.mark.parametrize("n,block", [c for c in CASES if c[1] == c[0] and c[0] <= 9000])
def test_gradient(solver, n, block):
    """L = sum lambda^3 / 3 = tr(T^3) / 3, so dL/dT = T^2 whatever basis the
    pairs' eigenvectors take; the repository's bar for gradients."""
    import torch

    d, e = _matrix(n, block)
    D, E = torch.tensor(d, device="cuda"), torch.tensor(e, device="cuda")
    ws = solver.new_checkpoint_workspace(n)
    W = solver.dstebr(D, E, workspace=ws)
    gD, gE = solver.dstebr_backward(D, E, W * W, workspace=ws, keep_forward=True)
    rd = d * d
    rd[:-1] += e * e
    rd[1:] += e * e
    re = 2.0 * e * (d[:-1] + d[1:])
    scale = max(np.abs(rd).max(), np.abs(re).max())
    assert np.abs(gD.cpu().numpy() - rd).max() < 1e-9 * scale
    assert np.abs(gE.cpu().numpy() - re).max() < 1e-9 * scale


@pytest.mark.parametrize("n,block", [c for c in CASES if c[0] <= 10000])
def test_vectors(solver, n, block):
    """The bars of the eigenvector tests (orthogonality 1e-11, residual 1e-12
    of the norm)."""
    import torch

    d, e = _matrix(n, block)
    D, E = torch.tensor(d, device="cuda"), torch.tensor(e, device="cuda")
    W, Z = solver.dstebr_vectors(D, E)
    assert torch.equal(W, solver.dstebr(D, E))
    TZ = D[:, None] * Z
    TZ[:-1] += E[:, None] * Z[1:]
    TZ[1:] += E[:, None] * Z[:-1]
    assert float((TZ - Z * W).abs().max()) < 1e-12 * float(W.abs().max())
    gram = Z.T @ Z
    gram.diagonal().sub_(1.0)
    assert float(gram.abs().max()) < 1e-11
