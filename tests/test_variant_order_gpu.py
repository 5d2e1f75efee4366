"""The chunk-kernel variant that runs where nothing is timed (MGB_AUTOTUNE=0, the
allocation-free forward, inside a capture) is not the slow one."""
import ctypes

import pytest

from magnus_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n,dims", [("plain", 3, (9, 10, 12, 15)), ("mixed", 3, (9, 10, 12)),
                                              ("plain", 8, (3, 6, 8)), ("mixed", 12, (3, 6, 7)), ("mixed", 4, (5, 6, 8))])
def test_untimed_variant_is_not_slow(precision, n, dims, cuda, monkeypatch):
    """One trajectory, the best of five passes: the untimed choice within a quarter of
    the fastest variant, forward and backward."""
    import torch
    monkeypatch.setenv("MGB_AUTOTUNE", "0")
    lib, S = _lib.load(), 4097
    f64 = precision == "plain"
    for d in dims:
        torch.manual_seed(d)
        A = torch.randn(S, d, d, device=cuda, dtype=torch.float64 if f64 else torch.float32) / d
        out, cot, dA = torch.empty_like(A[0]), torch.ones_like(A[0]), torch.empty_like(A)
        prob = _lib.make_problem(kind=0, dtype_code=_lib.DTYPE_F64 if f64 else _lib.DTYPE_F32,
                                 precision=_lib.PRECISION_CODES[precision], op=_lib.OP_SUM, integrator=0, n=n, samples=S,
                                 dim=d, t0=0.0, tf=1.0)
        one = lambda t: (ctypes.c_void_p * 1)(t.data_ptr())  # noqa: E731
        times = []
        for v in (None, 0, 1, 2, 3):
            monkeypatch.delenv("MGB_FORCE_VARIANT", raising=False)
            if v is not None:
                monkeypatch.setenv("MGB_FORCE_VARIANT", str(v))
            plan = ctypes.c_void_p()
            _lib.check(lib.mgb_plan_create(ctypes.byref(prob), 1, one(A), one(out), one(cot), one(dA), ctypes.byref(plan)))
            best = [1e9, 1e9]
            for _ in range(6):
                e = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
                stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
                e[0].record()
                _lib.check(lib.mgb_plan_forward(plan, stream))
                e[1].record()
                _lib.check(lib.mgb_plan_vjp(plan, stream))
                e[2].record()
                torch.cuda.synchronize()
                best = [min(b, x.elapsed_time(y)) for b, x, y in zip(best, e, e[1:])]
            _lib.check(lib.mgb_plan_destroy(plan))
            times.append(best)
        for k in range(2):
            assert times[0][k] <= 1.25 * min(t[k] for t in times), (d, times)
