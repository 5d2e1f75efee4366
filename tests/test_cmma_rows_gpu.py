"""The warp-MMA forward pass at d = 64 holds small rows and graded matrices to
their own size, as the three-piece kernel does (A is scaled per row, P per
column, and the second pieces apart)."""
import ctypes

import numpy as np
import pytest

import collapsed
from magnus_gb300 import _lib, workloads

pytestmark = pytest.mark.gpu

RULES = {"Boole": 4, "Simpson": 2, "Trapezoid": 2, "Riemann": 1}


@pytest.mark.parametrize("rule", list(RULES))
@pytest.mark.parametrize("form", ["rows", "similar"])
@pytest.mark.parametrize("variant", [0, 2])
def test_graded_elements(variant, form, rule, cuda, monkeypatch):
    """Every element within 3 products x 3 x 2^-22 (the pieces of A, of P, and
    the product left out) of FP64, relative to the same element formed from
    |A|.  rows: the rows of A fall to 2^-30; similar: D B D^-1 with D of
    2^-10..2^10."""
    import torch
    monkeypatch.setenv("MGB_FORCE_VARIANT", str(variant))
    lib = _lib.load()
    d, n, S, tf = 64, 4, 137 // RULES[rule] * RULES[rule] + 1, 1.0
    A = workloads.config0_samples(seed=5, d=d, samples=S)
    if form == "rows":
        A = A * 2.0 ** -np.rint(np.linspace(0, 30, d))[:, None]
    else:
        D = 2.0 ** np.rint(np.linspace(-10, 10, d))
        A = A * D[:, None] / D
    A = A.astype(np.float32)
    At, out = torch.tensor(A, device=cuda), torch.empty((n, d, d), device=cuda)
    prob = _lib.make_problem(kind=0, dtype_code=_lib.DTYPE_F32, precision=_lib.PRECISION_MIXED, op=_lib.OP_MANY,
                             integrator=_lib.INTEGRATOR_CODES[rule], n=n, samples=S, dim=d, t0=0.0, tf=tf, checkpoint_K=64)
    _lib.check(lib.mgb_forward(ctypes.byref(prob), At.data_ptr(), out.data_ptr(), None, None, None))
    torch.cuda.synchronize()
    A64 = A.astype(np.float64)
    T = [P[-1] for P in collapsed._levels(A64, n, tf / (S - 1), rule)]
    size = [P[-1] for P in collapsed._levels(np.abs(A64), n, tf / (S - 1), rule)]
    om, _, _ = collapsed._small_forward(T, n)
    Eb = [np.zeros((d, d)) for _ in range(n)]  # the terms' other factors, formed from the sizes
    for x, w in zip(*collapsed.gl_nodes(n)):
        D = [np.eye(d)]
        for k in range(1, n):
            D.append((1 - x) * sum(size[j] @ D[k - 1 - j] for j in range(k)))
        Eb = [e + w * v for e, v in zip(Eb, D)]
    got = out.cpu().numpy().astype(np.float64)
    for k in range(n):
        bound = size[0] if k == 0 else sum(size[j] @ Eb[k - j] for j in range(k + 1))
        assert (np.abs(got[k] - om[k]) <= 9 * 2.0 ** -22 * bound).all(), (k, np.max(np.abs(got[k] - om[k]) / bound))
