"""Plain form: running integrals stay local to a chunk (or a lane's run of it)
and the carried state is added where a value is used, so that increments below
the carried total's last place still add up."""
import ctypes

import numpy as np
import pytest

from magnus_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [2, 3, 16])
def test_small_increments_add_up(d, cuda, monkeypatch):
    """a(t) I with a = 1 over the first chunk and 0.3 last places of its integral
    per sample over the second, Riemann's rule.  dOmega_2 / dA_i for a cotangent C
    is dt (P_i + R_i - T) C = dt^2 a_i C, the difference of integrals of size T: its
    error is theirs, eight roundings at most (256 and more increments lost would
    be 77)."""
    import torch
    monkeypatch.setenv("MGB_FORCE_VARIANT", "0")
    K = 8192
    S, dt = 2 * K + 1, 1.0 / (2 * K)
    a = np.ones(S)
    a[K + 1:] = 0.3 * 2.0 ** -53 / dt
    A = a[:, None, None] * np.eye(d)
    cot = np.random.default_rng(d).uniform(0.5, 1.0, (d, d))
    At, ct = torch.tensor(A, device=cuda), torch.tensor(cot, device=cuda)
    dA = torch.empty_like(At)
    prob = _lib.make_problem(kind=0, dtype_code=_lib.DTYPE_F64, precision=_lib.PRECISION_PLAIN, op=_lib.OP_ONE,
                             integrator=_lib.INTEGRATOR_CODES["Riemann"], n=2, samples=S, dim=d, t0=0.0, tf=1.0, checkpoint_K=K)
    _lib.check(_lib.load().mgb_vjp(ctypes.byref(prob), At.data_ptr(), ct.data_ptr(), None, dA.data_ptr(), None))
    torch.cuda.synchronize()
    want = dt * dt * a[:, None, None] * cot
    err = np.abs(dA.cpu().numpy() - want)[K + 1:] / (dt * cot)
    assert err.max() <= 8 * 2.0 ** -53, err.max() * 2.0 ** 53
