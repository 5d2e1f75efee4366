"""One-shot calls from several threads, each on its own stream, and more of them
pending behind a busy stream than descriptors are kept for at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _samples(seed, S, d):
    import torch
    rng = np.random.default_rng(seed)
    t = np.linspace(0, 1, S).reshape(1, S, 1, 1)
    C = rng.standard_normal((3, 3, 1, d, d)) / np.sqrt(d)
    return torch.tensor(C[0] + C[1] * np.sin(2 * t) + C[2] * t, device="cuda", requires_grad=True)


def _passes(A, n, times):
    import torch
    from magnus_gb300.autograd import magnus
    got = []
    for _ in range(times):
        out = magnus(A, n, 0.0, 1.0, op="sum", integrator="Boole", precision="plain")
        got.append((out.detach(), torch.autograd.grad(out.sum(), A)[0]))
    return got


def test_threads_and_pending_calls(cuda):
    """Every pass equals the same call made alone, bit for bit."""
    import torch
    shapes = [(2, 257, 4), (3, 129, 3), (16, 65, 3), (8, 513, 2)]
    inputs = [_samples(k, S, d) for k, (d, S, _) in enumerate(shapes)]
    alone = [_passes(A, n, 1)[0] for A, (_, _, n) in zip(inputs, shapes)]
    torch.cuda.synchronize()
    results, errors = [None] * len(shapes), []

    def work(k):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                torch.cuda._sleep(100_000_000)  # some 50 ms: the calls queue up behind it
                results[k] = _passes(inputs[k], shapes[k][2], 40)
            stream.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for got, (out, dA) in zip(results, alone):
        for o, g in got:
            assert torch.equal(o, out) and torch.equal(g, dA)
