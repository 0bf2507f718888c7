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


def test_elementwise_operands_that_do_not_fit_are_refused(kernels):
    """One size is handed to the kernel for all arrays: none may be shorter, of another type or strided."""
    p, g, m, v, scalars, shadow = (torch.zeros(16) for _ in range(6))
    shadow = shadow.bfloat16()
    good = dict(param=p, grad=g, exp_avg=m, exp_avg_sq=v, scalars=scalars, shadow=shadow)
    bad = {"param": [p.double(), torch.zeros(32)[::2]], "grad": [g[:8], g.half()], "exp_avg": [m[:8], m.bfloat16(), torch.zeros(32)[::2]],
           "exp_avg_sq": [v[:8], v.double()], "shadow": [shadow[:8], p, torch.zeros(32).bfloat16()[::2]], "scalars": [scalars[:7], scalars.double()]}
    for name, values in bad.items():
        for value in values:
            with pytest.raises(ValueError) as e:
                elementwise.adamw_step_dev(**{**good, name: value})
            assert "cuda device" not in str(e.value), name
    counter = torch.zeros(1, dtype=torch.float64)
    for args in [(counter.float(), scalars), (counter, scalars[:7]), (counter, scalars.double())]:
        with pytest.raises(ValueError, match="step counter"):
            elementwise.adam_prepare(args[0], (1e-3, (0.9, 0.95), 1e-8, 0.1), args[1])
    with pytest.raises(RuntimeError, match="size"):
        elementwise.multi_copy(p, [(p[:8], g)])
    elementwise.multi_copy(p, [(p, torch.ones(1))])  # as copy_ does
    assert torch.equal(p, torch.ones(16)) and kernels.calls == []


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


def refused_calls(make, ids):
    """Calls whose operands do not fit together, or are not what the kernels read.  make(*shape) -> a bf16 tensor, ids(*shape) -> int64 zeros."""
    from tandem_b200 import ops

    x, w, b, r = make(40, 64), make(96, 64), make(96), make(40, 96)
    table, positions, text = make(50, 64), make(32, 64), ids(2, 16)
    return {
        "linear: wider input": (ValueError, lambda: ops.linear(make(40, 72), w, b)),
        "linear: narrower input": (ValueError, lambda: ops.linear(make(40, 56), w, b)),
        "linear: transposed weight": (ValueError, lambda: ops.linear(x, make(64, 96).t(), b)),
        "linear: 1-D weight": (ValueError, lambda: ops.linear(x, make(64), b)),
        "linear: short bias": (ValueError, lambda: ops.linear(x, w, make(88))),
        "linear: long bias": (ValueError, lambda: ops.linear(x, w, make(104))),
        "linear: residual of one row": (ValueError, lambda: ops.linear(x, w, b, residual=make(1, 96))),
        "linear: narrow residual": (ValueError, lambda: ops.linear(x, w, b, residual=make(40, 88))),
        "mlp: wider input": (ValueError, lambda: ops.mlp(make(40, 72), w, b, make(64, 96), make(64), x)),
        "mlp: second weight": (ValueError, lambda: ops.mlp(x, w, b, make(64, 88), make(64), x)),
        "mlp: first bias": (ValueError, lambda: ops.mlp(x, w, make(88), make(64, 96), make(64), x)),
        "mlp: second bias": (ValueError, lambda: ops.mlp(x, w, b, make(64, 96), make(56), x)),
        "mlp: residual of one row": (ValueError, lambda: ops.mlp(x, w, b, make(64, 96), make(64), make(1, 64))),
        "mlp: wide residual": (ValueError, lambda: ops.mlp(x, w, b, make(64, 96), make(64), r)),
        "layer_norm: short weight": (ValueError, lambda: ops.layer_norm(x, make(56), make(64))),
        "layer_norm: short bias": (ValueError, lambda: ops.layer_norm(x, make(64), make(56))),
        "residual_layer_norm: short weight": (ValueError, lambda: ops.residual_layer_norm(x, make(56), make(64))),
        "attention: columns left over": (ValueError, lambda: ops.causal_attention(make(1, 128, 385), 2)),
        "embedding: 32-bit ids": (TypeError, lambda: ops.embedding(text.int(), table, positions)),
        "embedding: host ids": (TypeError, lambda: ops.embedding(torch.zeros(2, 16, dtype=torch.int64), table, positions)),
        "embedding: positions": (ValueError, lambda: ops.embedding(ids(2, 33), table, positions)),
        "embedding: widths": (ValueError, lambda: ops.embedding(text, table, make(32, 56))),
        "embedding: 1-D table": (ValueError, lambda: ops.embedding(text, table, make(64))),
        "cross_entropy: 32-bit targets": (TypeError, lambda: ops.cross_entropy(r, ids(40).int())),
        "cross_entropy: host targets": (TypeError, lambda: ops.cross_entropy(r, torch.zeros(40, dtype=torch.int64))),
        "cross_entropy: too few targets": (ValueError, lambda: ops.cross_entropy(r, ids(39))),
        "cross_entropy: too many targets": (ValueError, lambda: ops.cross_entropy(r, ids(41))),
    }


@pytest.mark.parametrize("native", [True, False])
def test_operands_that_do_not_fit_are_refused(native, monkeypatch):
    """On tensors that only have the shape of CUDA tensors, so that nothing could be launched."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    if native and _lib.native() is None:
        pytest.skip("the native operators are not built")
    if not native:
        monkeypatch.setattr(_lib, "native", lambda: None)
    with FakeTensorMode(allow_non_fake_inputs=True):
        assert (_lib.direct(torch.empty(2, device="cuda")) is not None) == native
        calls = refused_calls(lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device="cuda"),
                              lambda *shape: torch.zeros(*shape, dtype=torch.int64, device="cuda"))
        for name, (kind, call) in calls.items():
            with pytest.raises(kind) as e:
                call()
            assert type(e.value) is kind, name
