"""k_box with boxes of 64, 128 and 256 poles against the per-level kernels,
which sum every pole directly: a weakly disordered chain whose merges keep
nearly all their rows (more than 8192 and, below the root, more than 16,384
poles), so that roots, Loewner weights and rows of each box size go into the
eigenvalues and gradients."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def chain():
    import torch

    n = 40000
    rng = np.random.default_rng(40000)
    return (n, torch.tensor(0.01 * rng.standard_normal(n), device="cuda"),
            torch.ones(n - 1, dtype=torch.float64, device="cuda"))


def _both(solver, call):
    """call() with the fused levels and with the per-level kernels."""
    tuning = solver.tuning()
    out = call()
    try:
        solver.set_tuning(fused_level_rows=0)
        return out, call()
    finally:
        solver.set_tuning(**tuning)


def test_eigenvalues(solver, chain):
    """16 eps of the norm a level, as test_box_gpu.py has it; 12 levels."""
    n, D, E = chain
    W, V = _both(solver, lambda: solver.dstebr(D, E).clone())
    assert float((W - V).abs().max()) <= 12 * 16 * EPS * float(W.abs().max())
    ws = solver.workspace(n)
    solver.dstebr(D, E, workspace=ws)
    level = solver.diagnostics(n, ws)["level"]
    assert any(8192 < lv["dd_after_max"] <= 16384 for lv in level)
    assert any(lv["dd_after_max"] > 16384 for lv in level[:-1])


def test_gradient(solver, chain):
    """L = tr(T^3) / 3 has dL/dT = T^2; the repository's bar for gradients."""
    n, D, E = chain
    ws = solver.new_checkpoint_workspace(n)

    def grads():
        W = solver.dstebr(D, E, workspace=ws)
        gD, gE = solver.dstebr_backward(D, E, W * W, workspace=ws, keep_forward=True)
        return gD.clone(), gE.clone()

    rD = D * D
    rD[:-1] += E * E
    rD[1:] += E * E
    rE = 2.0 * E * (D[:-1] + D[1:])
    bound = 1e-9 * float(rD.abs().max())
    for gD, gE in _both(solver, grads):
        assert float((gD - rD).abs().max()) <= bound
        assert float((gE - rE).abs().max()) <= bound
