"""The workspace pool of the one-shot calls is bounded and given back on request."""
import pytest

pytestmark = pytest.mark.gpu


def test_release_workspaces(cuda):
    """64 trajectories of d = 16 take 0.8 GB of workspace: at most 1 GiB stays after
    the call, and nothing after the release; calls work as before."""
    import torch
    from magnus_gb300 import device
    from magnus_gb300.autograd import magnus
    A = torch.randn(64, 8101, 16, 16, device=cuda, dtype=torch.float32) / 4
    call = lambda: magnus(A, 6, 0.0, 1.0, op="sum", integrator="Boole", precision="mixed")  # noqa: E731
    first = call()
    device.release_workspaces()
    free = torch.cuda.mem_get_info()[0]
    second = call()
    torch.cuda.synchronize()
    kept = free - torch.cuda.mem_get_info()[0]
    device.release_workspaces()
    left = free - torch.cuda.mem_get_info()[0]
    assert (256 << 20) <= kept <= (1 << 30) + (64 << 20), kept
    assert left <= 32 << 20, left
    assert torch.equal(first, second) and torch.equal(call(), first)
