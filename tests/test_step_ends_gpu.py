"""The kernels at the two ends of a step: the arrays arrive whole on both ways they can take, the barrier is zero behind them, and
a code reaches the host only when there is one."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 4, 1023, 4100, 16384, 16385, 60000])
def test_step_begin(n):
    from qwen25vl_lite.ops import kernels
    staging = torch.arange(1, 65537, dtype=torch.int32).pin_memory()
    ints = torch.zeros(65536, dtype=torch.int32, device="cuda")
    barrier = kernels._chain_buffers(ints.device)[1]
    barrier.fill_(77)
    kernels.step_begin(staging, ints, n)
    assert torch.equal(ints[:n].cpu(), staging[:n]) and int(barrier.abs().sum()) == 0
    assert int(ints[(n + 3) // 4 * 4:].abs().sum()) == 0


def test_step_end():
    from qwen25vl_lite.ops import kernels
    host = torch.full((1,), 5, dtype=torch.int32).pin_memory()
    device = torch.device("cuda", torch.cuda.current_device())
    kernels.step_end(device, host)
    torch.cuda.synchronize()
    assert int(host[0]) == 5                       # no code: nothing is written
    kernels.error_flag(device).fill_(9)
    kernels.step_end(device, host)
    torch.cuda.synchronize()
    assert int(host[0]) == 9
    kernels.reset_after_error(device)
