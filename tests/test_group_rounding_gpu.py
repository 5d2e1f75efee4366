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


@pytest.mark.parametrize("rule", ["Boole", "Simpson", "Trapezoid", "Riemann"])
@pytest.mark.parametrize("d", [3, 8, 24])
def test_error_of_few_samples(d, rule, cuda, monkeypatch):
    """The same roundings per sample (Boole: per block): the errors against FP64
    are no larger, up to the order of the products' sums (2 %)."""
    n, S, B = 4, 9, 512 if d < 24 else 64
    rng = np.random.default_rng(d)
    t = np.linspace(0, 1, S).reshape(1, S, 1, 1)
    C = rng.standard_normal((3, B, 1, d, d)) / np.sqrt(d)
    A = (C[0] + C[1] * t + C[2] * np.cos(5 * t)).astype(np.float32).astype(np.float64)
    cot = rng.standard_normal((B, d, d)).astype(np.float32).astype(np.float64)
    ref = [np.stack(x) for x in zip(*[(collapsed.forward(a, n, 0.0, 1.0, "sum", rule),
                                       collapsed.vjp(a, c, n, 0.0, 1.0, "sum", rule)) for a, c in zip(A, cot)])]
    here = _run(0, A, cot, n, rule, monkeypatch)
    per_sample = _run(1, A, cot, n, rule, monkeypatch)
    for name, x, y, r in zip(("out", "dA"), here, per_sample, ref):
        assert _error(x, r) <= 1.02 * _error(y, r), (name, _error(x, r), _error(y, r))


def _fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(np.float32)


def _in_fp32(A, n, rule):
    """Omega_1 + .. + Omega_n of (B, S, 2, 2) samples on [0, 1], the levels in FP32 with
    the running integral compensated per block: the 2 x 2 kernel's arithmetic."""
    S = A.shape[1]
    bs, u, w = {"Boole": (4, 90, [[1 / 2, 1 / 2], [1 / 3, 4 / 3, 1 / 3], [3 / 8, 9 / 8, 9 / 8, 3 / 8],
                                  [14 / 45, 64 / 45, 24 / 45, 64 / 45, 14 / 45]]),
                "Simpson": (2, 6, [[1 / 2, 1 / 2], [1 / 3, 4 / 3, 1 / 3]])}[rule]
    dt = 1.0 / (S - 1)
    step = u * 2.0 ** np.round(np.log2(dt / u))  # exact weights
    w = [[np.float32(x * step) for x in row] for row in w]
    f, T = A, []
    for j in range(n):
        P, base, lo = np.zeros_like(A), np.zeros_like(A[:, 0]), np.zeros_like(A[:, 0])
        for b in range(0, S - 1, bs):
            for r in range(1, bs + 1):
                s = lo
                for i in sorted(range(r + 1), key=lambda i: w[r - 1][i]):
                    s = _fma(f[:, b + i], w[r - 1][i], s)
                P[:, b + r] = base + s
            v = base + s
            bb = v - base
            lo = (base - (v - bb)) + (s - bb)
            base = v
        T.append((base.astype(np.float64) + lo) * (dt / step) ** (j + 1))
        f = np.stack([np.stack([_fma(A[..., r, 1], P[..., 1, c], A[..., r, 0] * P[..., 0, c]) for c in (0, 1)], -1)
                      for r in (0, 1)], -2)
    return np.stack([sum(collapsed._small_forward([t[b] for t in T], n)[0]) for b in range(A.shape[0])])


@pytest.mark.parametrize("rule", ["Boole", "Simpson"])
def test_error_of_few_2x2_samples(rule, cuda, monkeypatch):
    """The 2 x 2 kernel's error over 2048 trajectories of nine samples against
    that of the same arithmetic on the host: the same roundings in another order
    (8192 elements: 5 % is six standard deviations)."""
    n, S, B = 4, 9, 2048
    rng = np.random.default_rng(2)
    t = np.linspace(0, 1, S).reshape(1, S, 1, 1)
    C = rng.standard_normal((3, B, 1, 2, 2)) / np.sqrt(2)
    A = (C[0] + C[1] * t + C[2] * np.cos(5 * t)).astype(np.float32)
    A64 = A.astype(np.float64)
    ref = np.stack([collapsed.forward(a, n, 0.0, 1.0, "sum", rule) for a in A64])
    here, _ = _run(0, A64, np.ones((B, 2, 2)), n, rule, monkeypatch)
    err, host = np.linalg.norm(here - ref), np.linalg.norm(_in_fp32(A, n, rule) - ref)
    assert err <= 1.05 * host, (err, host)
