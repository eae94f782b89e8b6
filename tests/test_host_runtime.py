"""The host side of the device calls against a CUDA runtime that runs nothing
(fake_cuda.cpp): what they do when memory is short or a launch fails, and the
order in which they leave the work of several streams."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT
from nbgpu import NBG_ECUDA, NBG_EINVAL, NBG_ENOMEM, NBG_OK, NbgDesc, ServerOpts

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


def descs(*items):
    d = (NbgDesc * len(items))()
    for k, x in enumerate(items):
        d[k] = NbgDesc(*x)
    return ctypes.cast(d, ctypes.c_void_p), len(items), d


# 8.5M output limbs: six-prime residues and constants 604 MB (a square) or 906,
# FP64 transforms and twiddles 470 or 705
LIMBS = 4_250_000
SHORT = {"sqr_dev": 550, "mul_dev": 800, "mul_batch_dev": 1000, "batch_create": 800, "mul_batch": 920}


@pytest.mark.parametrize("call", SHORT)
def test_products_that_only_fit_as_fp64_passes(fake, call):
    n, L = LIMBS, fake
    host = [(ctypes.c_uint64 * k)() for k in (2 * n, n, n)] if call == "mul_batch" else []
    for h in host:
        h[len(h) - 1] = 1
    r, a, b = (ctypes.addressof(h) for h in host) if host else (R, A, B)

    def run():
        if call == "sqr_dev":
            return L.nbg_sqr_dev(R, A, n, None)
        if call == "mul_dev":
            return L.nbg_mul_dev(R, A, n, B, n, None)
        if call == "batch_create":
            bt = ctypes.c_void_p()
            rc = L.nbg_batch_create(*descs((R, A, B, n, n, 0, 0))[:2], ctypes.byref(bt))
            return rc
        if call == "mul_batch":
            return L.nbg_mul_batch(*descs((r, a, b, n, n, 0, 0))[:2])
        return L.nbg_mul_batch_dev(*descs((R, A, B, n, n, 0, 0), (R + (1 << 40), A, None, n // 2, n // 2, 0, 0))[:2], None)

    L.fake_limit(SHORT[call] * 1_000_000)
    counts(L)
    assert run() == NBG_OK
    w, f = counts(L)
    assert w == 0 and f > 0
    # with room for them, word products again
    L.fake_limit(ctypes.c_size_t(-1).value)
    assert run() == NBG_OK
    w, f = counts(L)
    assert w > 0 and f == 0
    # nothing fits: refused, and the next call works
    L.fake_limit(0)
    big = 3 * n
    assert L.nbg_sqr_dev(R, A, big, None) == NBG_ENOMEM
    L.fake_limit(ctypes.c_size_t(-1).value)
    assert L.nbg_sqr_dev(R, A, big, None) == NBG_OK


def test_host_product_with_little_device_memory(fake):
    # residues, constants and limbs (43 MB) fit 62 MB, the shared workspace (64 MB at least) does not
    n = 200_000
    r, a, b = ((ctypes.c_uint64 * k)() for k in (2 * n, n, n))
    a[n - 1] = b[n - 1] = 1
    fake.nbg_mul.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p, ctypes.c_int64]
    fake.fake_limit(62_000_000)
    assert fake.nbg_mul(ctypes.addressof(r), ctypes.addressof(a), n, ctypes.addressof(b), n) == NBG_OK


@pytest.mark.parametrize("call", ["one", "batch", "host", "host_batch"])
def test_failed_launch_leaves_the_workspace_ordered(fake, call):
    # a launch fails: what was launched before it may still use the shared
    # workspace, so the next call's kernels come after it, on whatever stream
    L, s1, s2 = fake, 0x100, 0x200
    sizes = (5000, 40_000, 70_000, 90_000, 1000)
    hosts = [[(ctypes.c_uint64 * k)() for k in (2 * n, n)] for n in sizes]
    for _, a in hosts:
        a[len(a) - 1] = 1

    def run():
        if call == "one":
            return L.nbg_mul_dev(R, A, 40_000, B, 30_000, s1)
        if call.startswith("host"):
            use = hosts if call == "host_batch" else hosts[:1]
            return L.nbg_mul_batch(*descs(*((ctypes.addressof(r), ctypes.addressof(a), None, len(a), len(a), 0, 0)
                                            for r, a in use))[:2])
        return L.nbg_mul_batch_dev(*descs(*((R + (k << 30), A, B, n, n, 0, 0) for k, n in enumerate(sizes)))[:2], s1)

    assert run() == NBG_OK
    counts(L)
    assert run() == NBG_OK
    launches = counts(L)[0]
    assert launches >= (8 if "batch" in call else 3)
    for k in range(launches):
        L.fake_fail_at(k)
        assert run() == NBG_ECUDA
        L.fake_mark()
        assert L.nbg_mul_dev(R, A, 50_000, B, 30_000, s2) == NBG_OK
        assert L.fake_unordered() == 0, k


@pytest.mark.parametrize("m,n,direct", [(1700, 1500, 0), (16_000, 14_000, 0), (20_000, 15_000, 3), (100_000, 90_000, 3),
                                        (250_000, 240_000, 3)])
def test_pageable_operands_of_one_product(fake, m, n, direct):
    # short operands and results go through pinned staging; longer ones are the
    # driver's to copy (staging them took up to 1.6 times as long)
    r, a, b = ((ctypes.c_uint64 * k)() for k in (m + n, m, n))
    a[m - 1] = b[n - 1] = 1
    p = (ctypes.c_void_p * 3)(*(ctypes.addressof(x) for x in (r, a, b)))
    fake.fake_copied.argtypes = [ctypes.c_void_p, ctypes.c_int]
    fake.fake_copied(p, 3)
    assert fake.nbg_mul_batch(*descs((p[0], p[1], p[2], m, n, 0, 0))[:2]) == NBG_OK
    assert fake.fake_copied(p, 3) == direct


@pytest.mark.parametrize("count,limbs,coarse", [(23, 1000, 0), (24, 1000, 1), (256, 9000, 1), (100, 25_000, 1),
                                                (600, 5000, 0), (256, 20_000, 0), (10_000, 9000, 0)])
def test_batches_take_few_lengths_while_launches_weigh_more(fake, count, limbs, coarse):
    # from 24 products on, up to 5M output limbs
    bt = ctypes.c_void_p()
    d = descs(*((R + (k << 24), A, B, limbs, limbs, 64 * limbs, 64 * limbs) for k in range(count)))
    assert fake.nbg_batch_create(*d[:2], ctypes.byref(bt)) == NBG_OK
    assert fake.fake_coarse() == coarse


@pytest.mark.parametrize("la,lb,k", [(20_000, 20_000, 20_000), (60_000, 3000, 40_000), (100_000, 90_000, 250_000)])
def test_low_product_copies_what_it_keeps(fake, la, lb, k):
    # straight to the caller's limbs; through a full product in a fresh buffer
    # 60,000 limbs took 320 us, 250 before the driver made that copy
    r, a, b = ((ctypes.c_uint64 * n)(*([7] * n)) for n in (k, la, lb))
    fake.nbg_mullo.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p, ctypes.c_int64,
                               ctypes.c_int64]
    fake.fake_copied.argtypes = [ctypes.c_void_p, ctypes.c_int]
    p = (ctypes.c_void_p * 1)(ctypes.addressof(r))
    fake.fake_copied(p, 1)
    assert fake.nbg_mullo(ctypes.addressof(r), ctypes.addressof(a), la, ctypes.addressof(b), lb, k) == NBG_OK
    assert fake.fake_copied(p, 1) == 1
    full = min(la, k) + min(lb, k)
    assert not any(r[full:])  # limbs above the product
    # a zero operand is refused as before
    z = (ctypes.c_uint64 * 1)()
    assert fake.nbg_mullo(ctypes.addressof(r), ctypes.addressof(a), la, ctypes.addressof(z), 1, k) == NBG_EINVAL
