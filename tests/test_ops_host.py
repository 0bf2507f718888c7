"""The operators' host side, on CPU: what they refuse before a kernel could be launched."""

import pytest
import torch

from tandem_b200.ops import elementwise, gemm


class Recorder:
    """Stands in for the kernel library."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args: self.calls.append(name) or 0


@pytest.fixture
def kernels(monkeypatch):
    """The library's calls are recorded, and the raw stream query answers as it does beside a GPU: device -1 is the current one."""
    recorder = Recorder()
    monkeypatch.setattr(elementwise, "cuda_lib", lambda: recorder)
    monkeypatch.setattr(gemm, "lib", lambda: recorder)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 0, raising=False)
    return recorder


def test_host_tensors_are_refused_before_a_launch(kernels):
    p, m, v, g = (torch.zeros(16) for _ in range(4))
    scalars = torch.zeros(8)
    calls = [lambda: elementwise.multi_copy(p, [(p, g)]), lambda: elementwise.adamw_step_dev(p, g, m, v, scalars),
             lambda: elementwise.adam_prepare(torch.zeros(1, dtype=torch.float64), (1e-3, (0.9, 0.95), 1e-8, 0.1), scalars),
             lambda: gemm.gemm(g.view(2, 8), p.view(2, 8), 2, 2, 8, 8, 8, False, False)]
    for call in calls:
        with pytest.raises(ValueError, match="cuda device"):
            call()
    assert set(kernels.calls) <= {"tb_gemm_workspace_bytes"}
