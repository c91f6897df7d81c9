"""Merges that keep many poles (k_box, csrc/brdc_box.cuh): near sums and
interpolated far sums against LAPACK, where boxes are ragged, straddle gaps
of the spectrum or have no far part."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-12  # of the norm, the repository's bar for eigenvalues


def _matrix(kind, n, rng):
    e = np.ones(n - 1)
    if kind == "toeplitz":  # poles crowd at both ends of the spectrum
        d = np.full(n, 2.0)
    elif kind == "bands":  # 8 bands with gaps between them
        d = 3.0 * np.cos(2 * np.pi * np.arange(n) / 8) + 1e-3 * rng.standard_normal(n)
    elif kind == "narrow":  # bands 1e-6 wide around far apart centres
        d = np.tile([0.0, 1.0, 5.0, 100.0], n // 4 + 1)[:n] + 1e-8 * rng.standard_normal(n)
        e *= 0.02
    else:  # weak disorder: irregular spacings, most poles kept
        d = 0.05 * rng.standard_normal(n)
    return d, e


@pytest.mark.parametrize("kind", ["toeplitz", "bands", "narrow", "disorder"])
@pytest.mark.parametrize("n", [1025, 1100, 2047, 2050, 4097, 9001])
def test_against_lapack(solver, kind, n):
    import scipy.linalg
    import torch

    d, e = _matrix(kind, n, np.random.default_rng(n))
    D, E = torch.tensor(d, device="cuda"), torch.tensor(e, device="cuda")
    W = solver.dstebr(D, E).cpu().numpy()
    assert solver.info(n) == 0
    ref = scipy.linalg.eigvalsh_tridiagonal(d, e)
    assert np.abs(W - ref).max() <= TOL * np.abs(ref).max()


def test_batch_uses_boxes_for_smaller_merges(solver):
    """A batch sends merges of more than 512 poles there: ragged orders."""
    import scipy.linalg
    import torch

    rng = np.random.default_rng(2)
    orders = [513, 600, 640, 777, 1023, 1024, 1300, 2100]
    off = np.concatenate([[0], np.cumsum(orders)])
    D, E = np.empty(off[-1]), np.zeros(off[-1])
    for b, n in enumerate(orders):
        D[off[b]:off[b + 1]], E[off[b]:off[b + 1] - 1] = _matrix(("toeplitz", "disorder")[b % 2], n, rng)
    W = solver.dstebr_batched(off, torch.tensor(D, device="cuda"), torch.tensor(E, device="cuda")).cpu().numpy()
    for b in range(len(orders)):
        lo, hi = off[b], off[b + 1]
        ref = scipy.linalg.eigvalsh_tridiagonal(D[lo:hi], E[lo:hi - 1])
        assert np.abs(W[lo:hi] - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("kind", ["bands", "narrow"])
def test_same_as_sweeps_over_all_poles(solver, kind):
    """The per-level kernels sum every pole directly; one step of rounding
    apart (16 eps of the norm) with the merge tree's 8 levels of them."""
    import torch

    n = 4500
    d, e = _matrix(kind, n, np.random.default_rng(5))
    D, E = torch.tensor(d, device="cuda"), torch.tensor(e, device="cuda")
    W = solver.dstebr(D, E).clone()
    tuning = solver.tuning()
    try:
        solver.set_tuning(fused_level_rows=0)
        V = solver.dstebr(D, E)
    finally:
        solver.set_tuning(**tuning)
    bound = 8 * 16 * np.finfo(float).eps * float(W.abs().max())
    assert float((W - V).abs().max()) <= bound
