"""The host side of the device calls against a CUDA runtime that runs nothing
(fake_cuda.cpp): what they do when memory is short or a launch fails, and the
order in which they leave the work of several streams."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT
from nbgpu import NBG_ECUDA, NBG_ENOMEM, NBG_OK, NbgDesc, ServerOpts

SRC = os.path.join(ROOT, "nativebigint.jl_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def build(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    srcs = [os.path.join(SRC, f) for f in ("engine.cpp", "api.cpp", "serve.cpp")]
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", f"-I{SRC}", f"-I{CUDA}/include", "-o", out,
                    os.path.join(ROOT, "tests", "fake_cuda.cpp"), *srcs, "-lpthread", "-ldl"], check=True)
    return out


@pytest.fixture
def fake(build, tmp_path):
    # a copy per test: a fresh engine
    path = str(tmp_path / "libfake.so")
    with open(build, "rb") as f, open(path, "wb") as g:
        g.write(f.read())
    L = ctypes.CDLL(path, mode=os.RTLD_LOCAL | os.RTLD_NOW)
    vp, i64 = ctypes.c_void_p, ctypes.c_int64
    L.nbg_mul_dev.argtypes = [vp, vp, i64, vp, i64, vp]
    L.nbg_sqr_dev.argtypes = [vp, vp, i64, vp]
    L.nbg_mul_batch_dev.argtypes = [vp, i64, vp]
    L.nbg_batch_create.argtypes = [vp, i64, ctypes.POINTER(vp)]
    L.nbg_mul_batch.argtypes = [vp, i64]
    L.nbg_server_create.argtypes = [vp, ctypes.POINTER(vp)]
    L.nbg_submit_dev.argtypes = [vp, vp, ctypes.POINTER(i64)]
    L.nbg_wait.argtypes = [vp, i64, i64]
    L.nbg_server_destroy.argtypes = [vp]
    L.fake_limit.argtypes = [ctypes.c_size_t]
    L.fake_used.restype = ctypes.c_size_t
    L.fake_fail_at.argtypes = [ctypes.c_long]
    assert L.nbg_init(0) == NBG_OK
    return L


def counts(L):
    w, f = ctypes.c_long(), ctypes.c_long()
    L.fake_counts(ctypes.byref(w), ctypes.byref(f))
    return w.value, f.value


# addresses that nothing reads: device operands and results far apart
R, A, B = 1 << 44, 2 << 44, 3 << 44


def serve(L, budget, limbs):
    opts, s, t = ServerOpts(budget, 0, 0, 0, 0), ctypes.c_void_p(), ctypes.c_int64()
    assert L.nbg_server_create(ctypes.byref(opts), ctypes.byref(s)) == NBG_OK
    d = NbgDesc(R, A, B, limbs, limbs, 64 * limbs, 64 * limbs)
    assert L.nbg_submit_dev(s, ctypes.byref(d), ctypes.byref(t)) == NBG_OK
    rc = L.nbg_wait(s, t, 20_000_000)
    L.nbg_server_destroy(s)
    return rc


@pytest.mark.parametrize("limbs,budget,word", [
    # 4.3M output limbs: 302 MB of residues, 235 MB of FP64 transforms
    (2_150_000, 320_000_000, True), (2_150_000, 270_000_000, False), (4_250_000, 520_000_000, False),
    (8_500_000, 1_000_000_000, False), (1_048_576, 130_000_000, True)])
def test_server_serves_what_fits_the_fp64_passes(fake, limbs, budget, word):
    # transforms over six primes take more memory than the FP64 ones: a request
    # that only the latter fit in the budget runs on them
    assert serve(fake, budget, limbs) == NBG_OK
    w, f = counts(fake)
    assert (w > 0) == word and (f > 0) == (not word)
    # and one that neither fits is refused
    assert serve(fake, 20_000_000, limbs) == NBG_ENOMEM
