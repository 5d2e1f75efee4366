"""Autotuner picks: by the load of the call, and for the VJP by its own times."""
import ctypes
import json

import numpy as np
import pytest

import oracle as O
from conftest import rel
from magnus_gb300 import _lib

pytestmark = pytest.mark.gpu


def _plan(d, B, S, n, precision, dtype):
    """(description, A, cot, out, dA) of B equal trajectories after a forward
    pass and a VJP through a plan."""
    import torch
    lib, f64 = _lib.load(), dtype == "float64"
    rng = np.random.default_rng(d)
    t = np.linspace(0, 1, S).reshape(1, S, 1, 1)
    C = rng.standard_normal((3, B, 1, d, d)) / np.sqrt(d)
    A, cot = (C[0] + C[1] * np.sin(2 * t) + C[2] * t).astype(dtype), rng.standard_normal((B, d, d)).astype(dtype)
    At, ct = torch.tensor(A, device="cuda"), torch.tensor(cot, device="cuda")
    out, dA = torch.empty_like(ct), torch.empty_like(At)
    prob = _lib.make_problem(kind=0, dtype_code=_lib.DTYPE_F64 if f64 else _lib.DTYPE_F32,
                             precision=_lib.PRECISION_CODES[precision], op=_lib.OP_SUM, integrator=0, n=n, samples=S, dim=d,
                             t0=0.0, tf=1.0)
    ptrs = lambda x: (ctypes.c_void_p * B)(*[y.data_ptr() for y in x])  # noqa: E731
    plan = ctypes.c_void_p()
    _lib.check(lib.mgb_plan_create((_lib.Problem * B)(*[prob] * B), B, ptrs(At), ptrs(out), ptrs(ct), ptrs(dA),
                                   ctypes.byref(plan)))
    buf = ctypes.create_string_buffer(lib.mgb_plan_describe(plan, None, 0))
    lib.mgb_plan_describe(plan, buf, len(buf))
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(lib.mgb_plan_forward(plan, stream))
    _lib.check(lib.mgb_plan_vjp(plan, stream))
    torch.cuda.synchronize()
    _lib.check(lib.mgb_plan_destroy(plan))
    return json.loads(buf.value.decode())["segments"][0], A, cot, out.cpu().numpy(), dA.cpu().numpy()


def test_a_small_call_does_not_decide_for_a_large_one(cuda, monkeypatch):
    monkeypatch.delenv("MGB_FORCE_VARIANT", raising=False)
    monkeypatch.setenv("MGB_AUTOTUNE", "1")
    tiny, *_ = _plan(24, 1, 9, 3, "mixed", "float32")
    large, *_ = _plan(24, 64, 2049, 3, "mixed", "float32")
    again, *_ = _plan(24, 64, 2049, 3, "mixed", "float32")
    assert len(large["tuned_ms"]) == 3 and large["tuned_ms"] != tiny["tuned_ms"]
    assert min(large["tuned_ms"]) > min(tiny["tuned_ms"])  # its own sample of chunks
    assert again["tuned_ms"] == large["tuned_ms"]          # cached


@pytest.mark.parametrize("d,precision,dtype,tol,variants", [(8, "plain", "float64", 1e-12, 3), (20, "plain", "float64", 1e-12, 3),
                                                            (12, "mixed", "float32", 1e-6, 4), (5, "mixed", "float64", 1e-6, 3)])
def test_vjp_has_its_own_pick(d, precision, dtype, tol, variants, cuda, monkeypatch):
    monkeypatch.delenv("MGB_FORCE_VARIANT", raising=False)
    monkeypatch.setenv("MGB_AUTOTUNE", "1")
    seg, A, cot, out, dA = _plan(d, 2, 1025, 4, precision, dtype)
    assert len(seg["vjp_ms"]) == variants and seg["vjp_ms"][seg["vjp_variant"]] == min(seg["vjp_ms"]), seg
    for a, c, o, g in zip(A.astype(np.float64), cot.astype(np.float64), out, dA):
        assert rel(o, O.forward(a, 4, 0.0, 1.0, "sum", "Boole")) <= tol
        assert rel(g, O.vjp(a, c, 4, 0.0, 1.0, "sum", "Boole")) <= tol


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("d", [9, 11, 12])
def test_tile_kernel_as_fourth_variant(d, dtype, cuda, monkeypatch):
    monkeypatch.setenv("MGB_FORCE_VARIANT", "3")
    for S, n in ((45, 4), (9, 1), (301, 5)):
        seg, A, cot, out, dA = _plan(d, 2, S, n, "mixed", dtype)
        assert seg["variant"] == seg["vjp_variant"] == 3
        for a, c, o, g in zip(A.astype(np.float64), cot.astype(np.float64), out, dA):
            assert rel(o, O.forward(a, n, 0.0, 1.0, "sum", "Boole")) <= 1e-6
            assert rel(g, O.vjp(a, c, n, 0.0, 1.0, "sum", "Boole")) <= 1e-6
