"""Rounding of the block rules in the small-matrix chunk kernels: trajectories
of a few samples, where a rule's own sums are most of the error, against the
level-major kernel, which compensates sample by sample."""
import ctypes

import numpy as np
import pytest

import collapsed
from magnus_gb300 import _lib

pytestmark = pytest.mark.gpu


def _run(variant, A, cot, n, rule, monkeypatch):
    """(out, dA) of a batch of float64 samples in the mixed form."""
    import torch
    monkeypatch.setenv("MGB_FORCE_VARIANT", str(variant))
    lib = _lib.load()
    B, S, d, _ = A.shape
    At, ct = torch.tensor(A, device="cuda"), torch.tensor(cot, device="cuda")
    out, dA = torch.empty((B, d, d), dtype=torch.float64, device="cuda"), torch.empty_like(At)
    prob = _lib.make_problem(kind=0, dtype_code=_lib.DTYPE_F64, precision=_lib.PRECISION_MIXED, op=_lib.OP_SUM,
                             integrator=_lib.INTEGRATOR_CODES[rule], n=n, samples=S, dim=d, t0=0.0, tf=1.0)
    ptrs = lambda t: (ctypes.c_void_p * B)(*[x.data_ptr() for x in t])  # noqa: E731
    probs = (_lib.Problem * B)(*[prob] * B)
    _lib.check(lib.mgb_forward_batched(probs, B, ptrs(At), ptrs(out), None, None))
    _lib.check(lib.mgb_vjp_batched(probs, B, ptrs(At), ptrs(ct), None, ptrs(dA), None))
    torch.cuda.synchronize()
    return out.cpu().numpy(), dA.cpu().numpy()


def _error(got, ref):
    """Root mean square over the batch of the relative Frobenius errors."""
    axes = tuple(range(1, ref.ndim))
    return np.sqrt(np.mean(((got - ref) ** 2).sum(axes) / (ref ** 2).sum(axes)))


@pytest.mark.parametrize("rule", ["Trapezoid", "Riemann"])
@pytest.mark.parametrize("d", [3, 8, 24])
def test_error_of_few_samples(d, rule, cuda, monkeypatch):
    """The same roundings per sample: the errors against FP64 are equal up to
    the order of the products' sums (2 %)."""
    n, S, B = 4, 9, 512 if d < 24 else 64
    rng = np.random.default_rng(d)
    t = np.linspace(0, 1, S).reshape(1, S, 1, 1)
    C = rng.standard_normal((3, B, 1, d, d)) / np.sqrt(d)
    A = (C[0] + C[1] * t + C[2] * np.cos(5 * t)).astype(np.float32).astype(np.float64)
    cot = rng.standard_normal((B, d, d)).astype(np.float32).astype(np.float64)
    ref = [np.stack(x) for x in zip(*[(collapsed.forward(a, n, 0.0, 1.0, "sum", rule),
                                       collapsed.vjp(a, c, n, 0.0, 1.0, "sum", rule)) for a, c in zip(A, cot)])]
    here, per_sample = _run(0, A, cot, n, rule, monkeypatch), _run(1, A, cot, n, rule, monkeypatch)
    for name, x, y, r in zip(("out", "dA"), here, per_sample, ref):
        assert _error(x, r) <= 1.02 * _error(y, r), (name, _error(x, r), _error(y, r))
