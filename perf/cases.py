"""The work that users of the eigensolver have it do, as measurable cases.

Every case names an entry of the Python API and the input it is given:

  plain    Solver.dstebr on device buffers (values only)
  host     Solver.dstebr_host on page-locked host buffers
  grad     brdc.autograd.eigvalsh_tridiagonal, forward and backward
  step     Solver.dstebr on a checkpointing workspace, then
           Solver.dstebr_backward: the forward and adjoint of a training loop
  batch    Solver.dstebr_batched over uneven orders
  fit      dstebr_batched and dstebr_batched_backward: one gradient step of
           the inverse-eigenvalue fit sum (W - target)^2
  vectors  Solver.dstebr_vectors

The inputs are the four families of the plain-solve configuration (uniform,
normal, Toeplitz, clustered: brdc/families.py), drawn on the GPU from the
seed.  A Toeplitz matrix has two numbers only, so its seed moves those.
"""
import math
import os
import random
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "ppopp27-brdc-ae_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import brdc  # noqa: E402
from brdc.autograd import eigvalsh_tridiagonal  # noqa: E402

FAMILIES = ("uniform", "normal", "toeplitz", "clustered")


def listed():
    return [
        # one small matrix inside somebody's outer loop: latency and launches
        {"name": "plain_normal_100", "entry": "plain", "family": "normal", "n": 100},
        # a moderate odd order
        {"name": "plain_uniform_1001", "entry": "plain", "family": "uniform", "n": 1001},
        # the artifact's smoke configuration
        {"name": "plain_normal_4096", "entry": "plain", "family": "normal", "n": 4096},
        # the headline configuration: the largest order of the plain solve
        {"name": "plain_uniform_65536", "entry": "plain", "family": "uniform", "n": 65536},
        # heavy deflation at a large odd order
        {"name": "plain_clustered_49151", "entry": "plain", "family": "clustered", "n": 49151},
        # little deflation: all the O(n^2) secular work is done
        {"name": "plain_toeplitz_16384", "entry": "plain", "family": "toeplitz", "n": 16384},
        # a host program with its matrix in page-locked memory
        {"name": "host_uniform_16384", "entry": "host", "family": "uniform", "n": 16384},
        # a differentiable layer in a torch program
        {"name": "grad_normal_4096", "entry": "grad", "family": "normal", "n": 4096},
        # the forward and adjoint of a training loop at its largest order
        {"name": "step_normal_65536", "entry": "step", "family": "normal", "n": 65536},
        # thousands of independent matrices of all four families
        {"name": "batch_4096", "entry": "batch", "family": "mixed", "count": 4096, "lo": 32, "hi": 8192},
        # one step of the batched inverse-eigenvalue fit
        {"name": "fit_1024", "entry": "fit", "family": "normal", "count": 1024, "lo": 64, "hi": 4096},
        # eigenvectors too
        {"name": "vectors_normal_4096", "entry": "vectors", "family": "normal", "n": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(("plain", "plain", "plain", "host", "grad", "step", "batch", "fit", "vectors"))
    if entry in ("plain", "host"):
        return {"entry": entry, "family": rng.choice(FAMILIES), "n": _log_int(rng, 17, 65536)}
    if entry == "grad":
        return {"entry": entry, "family": rng.choice(("uniform", "normal")), "n": _log_int(rng, 64, 16384)}
    if entry == "step":
        return {"entry": entry, "family": rng.choice(("uniform", "normal")), "n": _log_int(rng, 512, 65536)}
    if entry == "vectors":
        return {"entry": entry, "family": rng.choice(("uniform", "normal")), "n": _log_int(rng, 64, 6000)}
    if entry == "batch":
        hi = _log_int(rng, 256, 8192)
        return {"entry": entry, "family": rng.choice(FAMILIES[:2] + ("mixed",)), "count": _log_int(rng, 16, 2048),
                "lo": 32, "hi": hi}
    hi = _log_int(rng, 256, 4096)
    return {"entry": entry, "family": rng.choice(("uniform", "normal")), "count": _log_int(rng, 16, 1024), "lo": 64,
            "hi": hi}


# ---------------------------------------------------------------- inputs
def _orders(case):
    """Orders of the instances: log-uniform and fixed by the case, so that
    every seed has the same shape."""
    if "n" in case:
        return [int(case["n"])]
    rng = random.Random(1000003 * case["count"] + case["hi"])
    return [_log_int(rng, case["lo"], case["hi"]) for _ in range(case["count"])]


def _offsets(orders):
    off = [0]
    for n in orders:
        off.append(off[-1] + n)
    return off


def _families(case, count):
    return [FAMILIES[i % 4] for i in range(count)] if case["family"] == "mixed" else [case["family"]] * count


def _inputs(case, seed):
    """Packed D and E (the slot after an instance's last row is 0)."""
    orders = _orders(case)
    off = _offsets(orders)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kw = {"dtype": torch.float64, "device": "cuda"}
    total, count = off[-1], len(orders)
    fam = torch.tensor([FAMILIES.index(f) for f in _families(case, count)], device="cuda")
    sizes = torch.tensor(orders, device="cuda")
    inst = torch.repeat_interleave(torch.arange(count, device="cuda"), sizes)
    row = torch.repeat_interleave(fam, sizes)
    ud, ue = torch.rand(total, generator=gen, **kw), torch.rand(total, generator=gen, **kw)
    nd, ne = torch.randn(total, generator=gen, **kw), torch.randn(total, generator=gen, **kw)
    a = 1.0 + 2.0 * torch.rand(count, generator=gen, **kw)
    b = 0.5 + torch.rand(count, generator=gen, **kw)
    centre = 2.0 * torch.rand(count, 8, generator=gen, **kw) - 1.0
    pick = torch.randint(0, 8, (total,), generator=gen, device="cuda")
    D = torch.where(row == 0, ud, torch.where(row == 1, nd, torch.where(
        row == 2, a[inst], centre[inst, pick] + 1.0e-10 * nd)))
    E = torch.where(row == 0, ue, torch.where(row == 1, ne, torch.where(row == 2, b[inst], 1.0e-6 * ue)))
    E[torch.tensor(off[1:], device="cuda") - 1] = 0.0
    return off, D, E, gen


def prepare(case, seed):
    off, D, E, gen = _inputs(case, seed)
    entry, total = case["entry"], off[-1]
    s = {"entry": entry, "solver": brdc.Solver()}
    if "n" in case:
        E = E[:-1].clone()
    s.update(D=D, E=E, off=off)
    new = lambda m: torch.empty(m, dtype=torch.float64, device="cuda")  # noqa: E731
    if entry == "plain":
        s.update(W=new(total), ws=s["solver"].workspace(total))
    elif entry == "host":
        joint = torch.empty(2 * total - 1, dtype=torch.float64).pin_memory()
        joint[:total].copy_(D)
        joint[total:].copy_(E)
        s.update(D=joint[:total], E=joint[total:], W=torch.empty(total, dtype=torch.float64).pin_memory(),
                 ws=s["solver"].host_workspace(total))
    elif entry in ("grad", "step"):
        s["G"] = torch.randn(total, generator=gen, dtype=torch.float64, device="cuda")
        if entry == "grad":
            s.update(D=D.requires_grad_(True), E=E.requires_grad_(True))
        else:
            s.update(W=new(total), gD=new(total), gE=new(total), ws=s["solver"].checkpoint_workspace(total))
    elif entry == "batch":
        s.update(W=new(total), ws=s["solver"].batched_workspace(off))
    elif entry == "fit":
        ws = s["solver"].batched_workspace(off, True)
        # targets: the spectra of a second seeded batch of the same orders
        _, D2, E2, _ = _inputs(case, seed + 7919)
        target = s["solver"].dstebr_batched(off, D2, E2, workspace=ws)
        s.update(W=new(total), gD=new(total), gE=new(total), ws=ws, target=target)
    elif entry == "vectors":
        import ctypes

        nb = ctypes.c_size_t(0)
        brdc.load().brdc_dstebr_vectors_workspace_size(total, ctypes.byref(nb))
        s["ws"] = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    return s


def run(s):
    solver, entry = s["solver"], s["entry"]
    if entry == "plain":
        return solver.dstebr(s["D"], s["E"], W=s["W"], workspace=s["ws"])
    if entry == "host":
        return solver.dstebr_host(s["D"], s["E"], W=s["W"], workspace=s["ws"])
    if entry == "grad":
        W = eigvalsh_tridiagonal(s["D"], s["E"], solver)
        gD, gE = torch.autograd.grad(W, (s["D"], s["E"]), s["G"])
        return {"W": W, "gD": gD, "gE": gE}
    if entry == "step":
        W = solver.dstebr(s["D"], s["E"], W=s["W"], workspace=s["ws"])
        gD, gE = solver.dstebr_backward(s["D"], s["E"], s["G"], workspace=s["ws"], keep_forward=True,
                                        gD=s["gD"], gE=s["gE"])
        return {"W": W, "gD": gD, "gE": gE}
    if entry == "batch":
        return solver.dstebr_batched(s["off"], s["D"], s["E"], W=s["W"], workspace=s["ws"])
    if entry == "fit":
        W = solver.dstebr_batched(s["off"], s["D"], s["E"], W=s["W"], workspace=s["ws"])
        G = 2.0 * (W - s["target"])
        gD, gE = solver.dstebr_batched_backward(s["off"], s["D"], s["E"], G, workspace=s["ws"],
                                                keep_forward=True, gD=s["gD"], gE=s["gE"])
        return {"W": W, "gD": gD, "gE": gE}
    W, Z = solver.dstebr_vectors(s["D"], s["E"], workspace=s["ws"])
    # an eigenvector is its line: the sign is fixed by its largest entry, as
    # programs do that store or compare vectors
    top = Z.gather(0, Z.abs().argmax(0, keepdim=True))
    return {"W": W, "Z": Z * top.sign()}


# ---------------------------------------------------------------- work
def _pairs(family, n):
    """Pole-root pairs of a merge tree over n rows (per sweep): a merge of m
    rows keeps about m poles up to the family's saturation, beyond which the
    eigenvectors' localisation deflates the rest; Toeplitz keeps half."""
    top = {"uniform": 140, "normal": 90, "toeplitz": n, "clustered": 24}[family]
    share = {"uniform": 0.8, "normal": 0.8, "toeplitz": 0.5, "clustered": 0.5}[family]
    pairs, m = 0.0, 32
    while m < 2 * n:
        k = min(share * min(m, n), top)
        pairs += max(1.0, n / m) * k * k
        m *= 2
    return pairs


def work(case):
    """Bytes: every input read once, every output written once.  Flops: the
    leaves' 16-row eigenproblems (values and two rows, about 9 n^2 each) and,
    per pole-root pair, three secular sweeps of 8, a Loewner factor of 4 and
    a boundary-row term of 10; the adjoint and the vectors on top."""
    orders = _orders(case)
    fams = _families(case, len(orders))
    n = sum(orders)
    pairs = sum(_pairs(f, m) for f, m in zip(fams, orders))
    words, flops = 3 * n, 144.0 * n + 38.0 * pairs
    if case["entry"] in ("grad", "step", "fit"):
        words, flops = 6 * n, flops + 144.0 * n + 30.0 * pairs
    if case["entry"] == "vectors":
        words, flops = words + n * n, flops + 4.0 * n * n * math.log2(max(2, n))
    return {"bytes": 8 * words, "flops": flops}


# ---------------------------------------------------------------- 64 bits
def _sturm(orders, D, E):
    """Eigenvalues by bisection with Sturm counts, 31 interior points a
    round, every root of every instance at once; ascending per instance."""
    count, top = len(orders), max(orders)
    off = _offsets(orders)
    sizes = torch.tensor(orders, device="cuda")
    start = torch.tensor(off[:-1], device="cuda")
    inst = torch.repeat_interleave(torch.arange(count, device="cuda"), sizes)
    rank = torch.arange(off[-1], device="cuda") - start[inst]
    far = 1.0e30  # a row past an instance's end never counts
    d = torch.full((top, count), far, dtype=torch.float64, device="cuda")
    e2 = torch.full((top, count), 1.0e-300, dtype=torch.float64, device="cuda")
    d[rank, inst] = D
    e2[rank, inst] = torch.clamp(E * E, min=1.0e-300)
    e2 = torch.cat([torch.full_like(e2[:1], 1.0e-300), e2[:-1]])
    Ea = E.abs()
    Eb = torch.cat([Ea.new_zeros(1), Ea[:-1]])
    radius = Ea + Eb
    norm = (D.abs() + radius).max()
    lo = torch.full((off[-1],), -float(norm) * 1.0001, dtype=torch.float64, device="cuda")
    hi = -lo
    frac = torch.arange(1, 32, dtype=torch.float64, device="cuda")[:, None] / 32.0
    lone = count == 1
    for _ in range(11):
        x = lo + (hi - lo) * frac
        q, below = torch.ones_like(x), torch.zeros(x.shape, dtype=torch.int32, device="cuda")
        t = torch.empty_like(x)
        for j in range(top):
            dj, ej = (d[j], e2[j]) if lone else (d[j][inst], e2[j][inst])
            torch.sub(dj, x, out=t)
            torch.div(ej, q, out=q)
            torch.sub(t, q, out=q)
            below.add_(q < 0)
        # the first point with more than `rank` eigenvalues below it
        first = (below <= rank).sum(0, keepdim=True)
        ends = torch.cat([lo[None], x, hi[None]])
        lo, hi = ends.gather(0, first)[0], ends.gather(0, first + 1)[0]
    return 0.5 * (lo + hi)


def _dense(D, E):
    T = torch.diag(D)
    i = torch.arange(E.numel(), device="cuda")
    T[i, i + 1] = E
    T[i + 1, i] = E
    return torch.linalg.eigh(T)


def exact(case, seed):
    entry, orders = case["entry"], _orders(case)
    big, total = max(orders), sum(orders)
    off, D, E, gen = _inputs(case, seed)
    if entry in ("plain", "host", "batch"):
        if case["family"] == "toeplitz":
            n = orders[0]
            a, b = D[0], E[0] if n > 1 else D.new_zeros(())
            k = torch.arange(1, n + 1, dtype=torch.float64, device="cuda")
            W = a - 2.0 * b * torch.cos(k * math.pi / (n + 1))
        elif big * max(1.0, total / 16384) > 20000:
            return None
        else:
            W = _sturm(orders, D, E)
        return W.cpu() if entry == "host" else W
    if entry == "fit" or big > 4096:
        return None
    W, V = _dense(D, E[:-1])
    if entry == "vectors":
        top = V.gather(0, V.abs().argmax(0, keepdim=True))
        return {"W": W, "Z": V * top.sign()}
    G = torch.randn(total, generator=gen, dtype=torch.float64, device="cuda")
    return {"W": W, "gD": (V * V) @ G, "gE": 2.0 * (V[:-1] * V[1:]) @ G}
