"""The leaf solver (csrc/brdc_leaf.cuh): one eigenpair per lane, checked on
the host against its own definition, and leaves that do and do not take it
side by side on the GPU."""
import ctypes

import numpy as np
import pytest

EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def leaf(built_lib):
    import build as b

    lib = ctypes.CDLL(b.HOSTLIB)
    dp = ctypes.POINTER(ctypes.c_double)
    lib.brdc_host_leaf.argtypes = [ctypes.c_int, dp, dp, dp, dp, dp]

    def call(d, e):
        s = len(d)
        a = [np.ascontiguousarray(d, dtype=float), np.append(e, 0.0), np.zeros(16), np.zeros(256), np.zeros(4)]
        ok = lib.brdc_host_leaf(s, *(x.ctypes.data_as(dp) for x in a))
        return ok, a[2][:s], a[3][: s * s].reshape(s, s)

    return call


def _matrix(kind, s, rng):
    if kind == "toeplitz":  # ends cut, so that 0 is an eigenvalue on Gershgorin's bound
        d, e = np.full(s, 2.0), np.ones(s - 1)
        d[0] -= 1.0
        d[-1] -= 1.0
    elif kind == "weak":  # couplings far apart in size
        d, e = rng.uniform(-1, 1, s), 10.0 ** rng.uniform(-9, 0, s - 1)
        e[0] = 0.5
    else:
        d, e = rng.standard_normal(s), np.abs(rng.standard_normal(s - 1))
    scale = 2.0 ** -(np.floor(np.log2(max(np.abs(d).max(), e.max()))) + 1)
    return d * scale, e * scale


@pytest.mark.parametrize("kind", ["normal", "toeplitz", "weak"])
@pytest.mark.parametrize("s", [2, 3, 8, 9, 15, 16])
def test_pairs_are_an_orthonormal_decomposition(leaf, kind, s):
    rng = np.random.default_rng(s)
    for _ in range(1 if kind == "toeplitz" else 50):
        d, e = _matrix(kind, s, rng)
        ok, lam, V = leaf(d, e)
        T = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
        if not ok:  # only where eigenvalues are too close for it
            assert kind == "weak" and np.diff(np.linalg.eigvalsh(T)).min() < 1e-5
            continue
        # a dot product of 16 terms rounds by at most 16 eps, a residual by
        # four products of entries below 1
        assert np.abs(V @ V.T - np.eye(s)).max() <= 16 * EPS
        assert np.abs(T @ V.T - V.T * lam).max() <= 16 * EPS
        assert np.all(np.diff(lam) > 0)


def test_close_eigenvalues_are_refused(leaf):
    """Two pairs 1e-9 apart: the vectors would be orthogonal to 1e-7 only."""
    d = np.array([0.5, 0.25, -0.5, 0.5 + 1e-9])
    ok, _, _ = leaf(d, np.array([1e-12, 0.3, 1e-12]))
    assert not ok


@pytest.mark.gpu
@pytest.mark.parametrize("ckpt", [False, True])
def test_mixed_leaves(solver, ckpt):
    """Instances whose leaves the eigenpair solver takes, nearly diagonal
    ones and close pairs, in the same half-warp pairs and warps."""
    import scipy.linalg
    import torch

    rng = np.random.default_rng(4)
    orders = [1, 2, 3, 16, 17, 31, 32, 33, 64, 100, 16, 32, 500]
    off = np.concatenate([[0], np.cumsum(orders)])
    D, E = rng.standard_normal(off[-1]), rng.standard_normal(off[-1])
    for b in range(len(orders)):
        lo, hi = off[b], off[b + 1]
        if b % 3 == 1:
            E[lo + (hi - lo) // 2:hi] *= 1e-7  # the second half is nearly diagonal
        if b % 3 == 2 and hi - lo > 3:
            D[lo + 2], E[lo], E[lo + 1:lo + 3] = D[lo], 1e-12, 1e-13
    t = lambda v: torch.tensor(v, device="cuda")  # noqa: E731
    ws = solver.batched_workspace(off, True) if ckpt else None
    W = solver.dstebr_batched(off, t(D), t(E), workspace=ws).cpu().numpy()
    for b in range(len(orders)):
        lo, hi = off[b], off[b + 1]
        ref = scipy.linalg.eigvalsh_tridiagonal(D[lo:hi], E[lo:hi - 1])
        assert np.abs(W[lo:hi] - ref).max() <= 1e-12 * np.abs(ref).max()
