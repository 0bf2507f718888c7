"""The host code of the kernel library without a GPU: its objects are linked against a CUDA runtime that takes launches down
instead of executing them (native/fake_cuda.cpp)."""

import ctypes
import os
import shutil
import subprocess

import pytest

from tandem_b200.utils import build

HERE = os.path.dirname(os.path.abspath(__file__))
I, P, LL = ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong
WORK = P(1 << 20)  # an address that nothing follows, aligned


def signatures(lib):
    lib.tb_gemm_bf16.argtypes = [P, P, P, I, I, I, I, I, I, I, I, I, P, P, P, I, P, LL, P]
    lib.tb_gemm_workspace_bytes.argtypes, lib.tb_gemm_workspace_bytes.restype = [I, I, I], LL
    lib.tb_col_sum.argtypes = [P, I, I, I, P, P, P]
    lib.tb_layernorm_bwd_add.argtypes = [P] * 10 + [I, I, P]
    lib.tb_attn_fwd.argtypes = [P, P, P, I, I, I, I, P]
    lib.tb_attn_bwd.argtypes = [P] * 6 + [I, I, I, I, P]
    return lib


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if shutil.which("g++") is None or build.nvcc_path() is None:
        pytest.skip("no compiler")
    objs = [o for o in build.cuda_objects() if os.path.basename(o) in ("gemm.o", "layers.o", "attention.o")]
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    # -Bsymbolic: its own runtime, not one that torch may have brought into the process
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-Wl,--no-undefined", f"-I{build.cuda_include()}", f"-I{build.CUDA}",
                        os.path.join(HERE, "native", "fake_cuda.cpp"), *objs, "-o", out, "-lpthread"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return signatures(ctypes.CDLL(out))


@pytest.mark.parametrize("products", [0, 1])
def test_threads_never_share_words(fake, products):
    """Tickets of column sums and flags of split products are handed out in turn, so every place of the pool is lent equally often,
    whatever the threads' timing.  A place lent twice in a round (two launches in flight would use the same words) is missing elsewhere."""
    out = (ctypes.c_ulonglong * 5)()  # places, lent at least, lent at most, first, last
    fake.fake_borrowed(out)
    threads, each = 8, 20000
    assert fake.fake_threads(threads, each, products) == 0
    fake.fake_borrowed(out)
    assert out[0] > 50 and out[0] * out[1] <= threads * each <= out[0] * out[2]
    assert out[2] - out[1] <= 1, f"{out[0]} places, lent {out[1]} to {out[2]} times"


@pytest.mark.parametrize("products", [0, 1])
def test_recorded_launches_keep_their_words(fake, products):
    """A graph's launches use theirs at every replay: none is lent to a launch that is not recorded, however many follow."""
    out, ranges = (ctypes.c_ulonglong * 5)(), {}
    fake.fake_borrowed(out)
    for recorded in (0, 1, 0, 1):
        fake.fake_record(recorded)
        assert fake.fake_threads(1, 5000, products) == 0
        fake.fake_borrowed(out)
        assert ranges.setdefault(recorded, (out[3], out[4])) == (out[3], out[4])
    fake.fake_record(0)
    assert ranges[0][1] < ranges[1][0]


def launches(lib):
    """A call of each kind that needs more than 48 KB of shared memory: (name, function)."""
    def product(M, N, K):
        need = lib.tb_gemm_workspace_bytes(M, N, K)
        return lib.tb_gemm_bf16(WORK, WORK, WORK, M, N, K, M, N, N, 1, 1, 0, None, None, None, 0, WORK if need else None, need, None)

    yield "product of few tiles", lambda: product(256, 256, 256)
    yield "product of pair tiles", lambda: product(8192, 4096, 512)
    for D in (256, 768, 1024, 1536, 2048):
        for add in (None, WORK):
            yield f"layer norm {D} {add}", lambda D=D, add=add: lib.tb_layernorm_bwd_add(*[WORK] * 5, add, *[WORK] * 4, 30000, D, None)
    for hd in (64, 128):
        for batch in (1, 64):
            yield f"attention {hd} {batch}", lambda hd=hd, batch=batch: (lib.tb_attn_fwd(WORK, WORK, WORK, batch, 1024, 8, hd, None)
                                                                      or lib.tb_attn_bwd(*[WORK] * 6, batch, 1024, 8, hd, None))


def test_shared_memory_is_allowed_on_every_device(fake):
    """The limit belongs to a device: a process that turns to a second one raises it there, too."""
    for device in (0, 1, 63, 64, 0):
        fake.fake_set_device(device)
        for name, call in launches(fake):
            assert call() == 0, (name, device)
    fake.fake_set_device(0)


def test_a_refused_limit_is_asked_for_again(fake):
    for device, (name, call) in enumerate(launches(fake), start=8):  # some share a kernel: each has a device of its own
        fake.fake_set_device(device)
        fake.fake_refuse_allowing(1)
        assert call() != 0, name
        fake.fake_refuse_allowing(0)
        assert call() == 0, name
    fake.fake_set_device(0)
