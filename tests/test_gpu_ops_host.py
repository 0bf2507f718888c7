"""The operators' host side on a GPU machine, over a kernel library that launches nothing (native/fake_kernels.cpp)."""

import ctypes
import os
import subprocess

import pytest
import torch

from tandem_b200.ops import _lib, gemm
from tandem_b200.utils import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake_path(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libfake_kernels.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", f"-I{build.CUDA}", f"-I{build.cuda_include()}", os.path.join(HERE, "native", "fake_kernels.cpp"), "-o", out], check=True)
    return out


@pytest.fixture(params=["native", "python"])
def kernels(request, fake_path, monkeypatch):
    fake = ctypes.CDLL(fake_path)
    fake.tb_gemm_last_error.restype = ctypes.c_char_p
    fake.tb_gemm_workspace_bytes.restype = ctypes.c_longlong
    fake.tb_stream_wait.argtypes = [ctypes.c_void_p] * 2
    torch.zeros(1, device="cuda")
    if request.param == "native":
        _lib.native().bind(fake_path)
    else:
        monkeypatch.setattr(_lib, "native", lambda: None)
        monkeypatch.setattr(_lib, "lib", lambda: fake)
        monkeypatch.setattr(gemm, "lib", lambda: Untyped(fake))
    yield fake
    if request.param == "native":
        _lib.native().bind(build.CUDA_LIB)


class Untyped:
    """The Python operators pass pointers as numbers, which a function without argument types would cut to 32 bits."""

    def __init__(self, fake):
        self.fake = fake

    def __getattr__(self, name):
        f = getattr(self.fake, name)
        return lambda *args: f(*(ctypes.c_void_p(a) if isinstance(a, int) and abs(a) >= 1 << 31 else a for a in args))


def leaf(*shape):
    return torch.zeros(*shape, dtype=torch.bfloat16, device="cuda", requires_grad=True)


def waits(fake):
    n = ctypes.c_int.in_dll(fake, "fake_waits")
    log = (ctypes.c_void_p * 2 * 64).in_dll(fake, "fake_log")
    out = [tuple(log[i]) for i in range(n.value)]
    n.value = 0
    return out


@pytest.mark.parametrize("name,launches", [("linear", 3), ("mlp", 6)])
def test_a_refused_launch_leaves_no_branch(name, launches, kernels):
    """Whichever launch of backward is refused: the second stream has been joined again by the time the error arrives."""
    from tandem_b200 import ops

    make = {"linear": lambda: ops.linear(leaf(40, 64), leaf(96, 64), leaf(96)),
            "mlp": lambda: ops.mlp(leaf(40, 64), leaf(96, 64), leaf(96), leaf(64, 96), leaf(64), leaf(40, 64))}[name]
    fail_at = ctypes.c_int.in_dll(kernels, "fake_fail_at")
    for at in range(1, launches + 2):
        y = make()
        waits(kernels)
        fail_at.value = at
        if at <= launches:
            with pytest.raises(RuntimeError, match="-77"):
                y.backward(torch.ones_like(y))
        else:  # one more than there are: every launch has been counted
            y.backward(torch.ones_like(y))
            assert fail_at.value == 1
        fail_at.value = 0
        log = waits(kernels)
        assert log and len(log) % 2 == 0
        for fork, join in zip(log[::2], log[1::2]):
            assert fork[::-1] == join, (at, log)


CALLS = {
    "linear": lambda ops: ops.linear(leaf(40, 64), leaf(96, 64), leaf(96)),
    "mlp": lambda ops: ops.mlp(leaf(40, 64), leaf(96, 64), leaf(96), leaf(64, 96), leaf(64), leaf(40, 64)),
    "layer_norm": lambda ops: ops.layer_norm(leaf(40, 64), leaf(64), leaf(64)),
    "residual_layer_norm": lambda ops: ops.residual_layer_norm(leaf(40, 64), leaf(64), leaf(64)),
    "causal_attention": lambda ops: ops.causal_attention(leaf(1, 128, 192), 1),
    "embedding": lambda ops: ops.embedding(torch.zeros(2, 8, dtype=torch.int64, device="cuda"), leaf(50, 64), leaf(32, 64)),
    "cross_entropy": lambda ops: ops.cross_entropy(leaf(40, 64), torch.zeros(40, dtype=torch.int64, device="cuda")),
}


@pytest.mark.parametrize("gradients", [True, False])
@pytest.mark.parametrize("name", CALLS)
def test_a_launch_that_waits_stops_no_other_thread(name, gradients, kernels):
    """A launch waits where the queue is full: the interpreter goes on meanwhile, here the thread that ends the wait."""
    import threading
    import time

    from tandem_b200 import ops

    closed = ctypes.c_int.in_dll(kernels, "fake_closed")
    started = threading.Event()

    def open_up():
        started.wait()
        time.sleep(0.05)
        closed.value = 0

    other = threading.Thread(target=open_up)
    other.start()
    with torch.set_grad_enabled(gradients):
        closed.value = 1
        started.set()
        CALLS[name](ops)  # ends with an error (-78) if nobody opens up
    other.join()
