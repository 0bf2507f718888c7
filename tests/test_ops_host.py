"""The operators' host side, on CPU: what they refuse before a kernel could be launched."""

import importlib.util

import pytest
import torch

from tandem_b200.ops import _lib, elementwise, gemm


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
    monkeypatch.setattr(_lib, "_raw_stream", lambda device: 0)
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


class Probe(torch.autograd.Function):
    """Tells whether a call went through the node (whose context torch makes) or through the forward alone."""

    @staticmethod
    def forward(ctx, x):
        Probe.bare = isinstance(ctx, Probe.untracked)
        return x * 2


@pytest.mark.parametrize("missing", [None, "_get_tracing_state", "_functorch", "_cuda_getCurrentRawStream", "_current_level"])
def test_torch_without_an_undocumented_name(missing, monkeypatch):
    """The forward alone is called where gradients are off, and only if torch can tell that nothing else wants the node."""
    if missing is not None:
        monkeypatch.delattr(torch.autograd.forward_ad if missing == "_current_level" else torch._C, missing)
    spec = importlib.util.spec_from_file_location("tandem_b200.ops._lib_again", _lib.__file__)
    again = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(again)
    monkeypatch.undo()
    Probe.untracked = again._Untracked
    x = torch.ones(3)
    with torch.no_grad():
        assert torch.equal(again.run(Probe, x), x * 2)
        assert Probe.bare == (missing in (None, "_cuda_getCurrentRawStream"))
        if Probe.bare:
            torch.jit.trace(lambda v: again.run(Probe, v), x, check_trace=False)
            assert not Probe.bare
    again.run(Probe, x)
    assert not Probe.bare
