"""mgb_plan_describe names the kernels that run."""
import ctypes
import json

import pytest

from magnus_gb300 import _lib

pytestmark = pytest.mark.gpu

M, P = _lib.PRECISION_MIXED, _lib.PRECISION_PLAIN


@pytest.mark.parametrize("d,n,precision,variant,forward,vjp,ctas,scan", [
    (2, 4, M, 0, "k_small", "k_small", 0, "per-instance"),
    (8, 4, P, 0, "k_col", "k_col", 0, "per-instance"),
    (8, 4, P, 1, "k_chunk", "k_chunk", 4, "per-instance"),
    (20, 4, P, 0, "k_dense", "k_dense", 0, "per-instance"),
    (12, 4, M, 3, "k_dense", "k_dense", 0, "per-instance"),
    (12, 4, M, 0, "k_chunk", "k_chunk", 8, "per-instance"),
    (16, 4, M, 0, "k_tile", "k_tile", 2, "columns"),
    (16, 4, P, 1, "k_chunk", "k_chunk", 4, "tiled"),
    (32, 4, M, 2, "k_tiletc", "k_mma32", 2, "columns"),
    (32, 4, M, 3, "k_cmma", "k_mma32", 4, "columns"),
    (32, 7, M, 0, "k_tile", "k_tile", 2, "per-instance"),
    (64, 4, M, 2, "k_cmma", "k_bigtc", 1, "columns"),
    (64, 4, M, 4, "k_bigtc", "k_bigtc", 3, "columns"),
    (64, 7, M, 1, "k_bigtc", "k_bigtc", 2, "tiled"),
])
def test_kernel_names(d, n, precision, variant, forward, vjp, ctas, scan, cuda, monkeypatch):
    import torch
    monkeypatch.setenv("MGB_FORCE_VARIANT", str(variant))
    lib, dt = _lib.load(), torch.float32 if precision == M else torch.float64
    A = torch.zeros(33, d, d, device=cuda, dtype=dt)
    out, dA = torch.empty_like(A[0]), torch.empty_like(A)
    prob = _lib.make_problem(kind=0, dtype_code=_lib.DTYPE_F32 if precision == M else _lib.DTYPE_F64, precision=precision,
                             op=_lib.OP_SUM, integrator=0, n=n, samples=33, dim=d, t0=0.0, tf=1.0)
    one = lambda t: (ctypes.c_void_p * 1)(t.data_ptr())  # noqa: E731
    plan = ctypes.c_void_p()
    _lib.check(lib.mgb_plan_create(ctypes.byref(prob), 1, one(A), one(out), one(out), one(dA), ctypes.byref(plan)))
    buf = ctypes.create_string_buffer(lib.mgb_plan_describe(plan, None, 0))
    lib.mgb_plan_describe(plan, buf, len(buf))
    _lib.check(lib.mgb_plan_destroy(plan))
    seg = json.loads(buf.value.decode())["segments"][0]
    assert (seg["forward"], seg["vjp"], seg["ctas_per_sm"], seg["scan"]) == (forward, vjp, ctas, scan), seg
