"""Runs per chunk of the column kernel (d = 3..8): the CTA that launches holds
a chunk's runs at every size, and the largest counts match the oracle."""
import ctypes

import numpy as np
import pytest

import oracle as O
from conftest import rel
from magnus_gb300 import _lib


def _symbol(name, *argtypes, restype=ctypes.c_int):
    f = getattr(_lib.load(), name)
    f.argtypes, f.restype = argtypes, restype
    return f


@pytest.mark.parametrize("plain", [False, True])
@pytest.mark.parametrize("d", [3, 4, 5, 6, 7, 8])
def test_runs_fit_the_cta(d, plain):
    """mgb::col_lanes against the teams of the CTA it selects (32 / d a warp;
    64 threads, 128 in the plain form with sixteen runs), and the scratch sizes
    that follow from it (mgb::col_scratch, mgb::col_scratch_min)."""
    i32, i64 = ctypes.c_int, ctypes.c_int64
    lanes = _symbol("_ZN3mgb9col_lanesEbiilli", ctypes.c_bool, i32, i32, i64, i64, i32)
    scratch = _symbol("_ZN3mgb11col_scratchEbiillii", ctypes.c_bool, i32, i32, i64, i64, i32, i32, restype=i64)
    least = _symbol("_ZN3mgb15col_scratch_minEbiili", ctypes.c_bool, i32, i32, i64, i32, restype=i64)
    for sms in (1, 148, 152):
        for n in (1, 2, 3, 4, 5, 6, 8, 12):
            for nwork in (1, 2, 16, 100, 197, 1000, 100000):
                for kmax in (1, 4, 35, 252, 253, 256, 512, 1024, 1 << 20):
                    runs = lanes(plain, d, n, nwork, kmax, sms)
                    teams = 32 // d * (4 if plain and runs == 16 else 2)
                    assert 1 <= runs <= teams, (sms, n, nwork, kmax, runs)
                    assert scratch(plain, d, n, nwork, kmax, runs, sms) >= least(plain, d, n, kmax, runs) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,d", [("float64", 3), ("float64", 4), ("complex128", 2)])
def test_most_runs_match_oracle(dtype, d, cuda):
    """Few chunks at low orders (n = 1, 2 at the default interval, 3, 4 at 512
    samples), where the run count is the largest: the plain form's 1e-12."""
    import torch
    from magnus_gb300.autograd import magnus
    rng = np.random.default_rng(d)
    z = (lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)) if dtype == "complex128" else \
        (lambda *s: rng.standard_normal(s))
    for rule, intervals, K, n in (("Boole", 256, 0, 1), ("Simpson", 512, 0, 2), ("Riemann", 257, 0, 2),
                                  ("Boole", 1024, 512, 3), ("Trapezoid", 510, 512, 4)):
        t = np.linspace(0, 1, intervals + 1).reshape(-1, 1, 1)
        C = z(3, 1, d, d) / np.sqrt(d)
        A = (C[0] + C[1] * np.sin(2 * t) + C[2] * t).astype(dtype)
        cot = z(d, d).astype(dtype)
        At = torch.tensor(A, device=cuda, requires_grad=True)
        out = magnus(At, n, 0.0, 1.0, op="sum", integrator=rule, precision="plain", checkpoint_K=K)
        g, = torch.autograd.grad(out, At, torch.tensor(cot, device=cuda))
        if dtype == "complex128":  # [[Re, -Im], [Im, Re]]
            E = np.concatenate([np.concatenate([A.real, -A.imag], 2), np.concatenate([A.imag, A.real], 2)], 1)
            ref = O.forward(E, n, 0.0, 1.0, "sum", rule)
            dE = O.vjp(E, np.block([[cot.real, 0 * cot.real], [cot.imag, 0 * cot.real]]), n, 0.0, 1.0, "sum", rule)
            ref = ref[:d, :d] + 1j * ref[d:, :d]
            gref = dE[:, :d, :d] + dE[:, d:, d:] + 1j * (dE[:, d:, :d] - dE[:, :d, d:])
        else:
            ref, gref = O.forward(A, n, 0.0, 1.0, "sum", rule), O.vjp(A, cot, n, 0.0, 1.0, "sum", rule)
        assert rel(out.detach().cpu().numpy(), ref) <= 1e-12, (rule, n)
        assert rel(g.cpu().numpy(), gref) <= 1e-12, (rule, n)
