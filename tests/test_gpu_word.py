"""Products through the five-prime word transforms (one 64-bit limb per
coefficient): every transform shape at its exact length and one below, values
whose coefficients and carries are extreme, and mixed batches, all equal to
GMP's product and to the FP64 passes' (integers: no tolerance)."""
import json

import numpy as np
import pytest

import oracle as O
from conftest import adversarial, rand_limbs

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# (odd multiplier, log2 of the rest): each column-pass and block variant, the
# smallest and largest lengths of the range
SHAPES = [(1, 6), (3, 8), (5, 9), (7, 8), (1, 7), (1, 8), (1, 9), (1, 10), (1, 11), (1, 12), (1, 13), (1, 14), (1, 15), (1, 16), (1, 17),
          (3, 6), (3, 7), (3, 9), (3, 10), (3, 12), (3, 13), (3, 14), (3, 15),
          (5, 6), (5, 7), (5, 8), (5, 12), (5, 13), (5, 14),
          (7, 6), (7, 7), (7, 10), (7, 12), (7, 13), (7, 14),
          # two column passes
          (1, 18), (1, 19), (1, 20), (3, 16), (3, 17), (3, 18), (3, 20), (5, 15), (5, 16), (5, 17), (5, 19),
          (7, 15), (7, 16), (7, 18), (7, 19)]


def _want(a, b):
    return O.gmp_sqr(a) if b is None else O.gmp_mul(a, b)


def _kinds(nbgpu, a, b):
    da, db = torch.from_numpy(a).cuda(), None if b is None else torch.from_numpy(b).cuda()
    r = torch.zeros(a.size + (a.size if b is None else b.size), dtype=torch.uint64, device="cuda")
    bits = [64 * x.size for x in (a, a if b is None else b)]
    bt = nbgpu.Batch(nbgpu.make_descs([(r, da, db, a.size, r.numel() - a.size, *bits)]))
    kinds = {s["kind"] for s in bt.stats()}
    bt.close()
    return kinds


@pytest.mark.parametrize("odd,k", SHAPES)
def test_word_shapes(gpu_lib, odd, k):
    N = odd << k
    rng = np.random.default_rng(N)
    for n1 in (N + 1, N):  # m + n - 1 = N and N - 1 coefficients
        n = n1 * 2 // 5
        a, b = rand_limbs(rng, n1 - n), rand_limbs(rng, n)
        assert np.array_equal(gpu_lib.mul(a, b), _want(a, b))
        # the largest coefficients and a carry through every limb
        ones = np.full(n1 - n, 2**64 - 1, dtype=np.uint64)
        assert np.array_equal(gpu_lib.mul(ones, ones[:n].copy()), _want(ones, ones[:n].copy()))
    s = rand_limbs(rng, (N + 1) // 2)
    assert np.array_equal(gpu_lib.sqr(s), _want(s, None))


def test_word_kernels_run_and_edge_operands(gpu_lib):
    rng = np.random.default_rng(77)
    a, b = rand_limbs(rng, 3000), rand_limbs(rng, 2500)
    assert "k_wsmall" in _kinds(gpu_lib, a[:200].copy(), b[:100].copy())
    assert "k_wtail" in _kinds(gpu_lib, a, b) and "k_wtail" in _kinds(gpu_lib, a, None)
    for m, n in ((1, 1), (2, 1), (700, 1), (513, 512), (65536, 65537), (130000, 3)):
        x, y = adversarial(rng, m), adversarial(rng, n)
        assert np.array_equal(gpu_lib.mul(x, y), _want(x, y))
    z = np.zeros(4096, dtype=np.uint64)  # zero limbs above the magnitude
    z[:3] = rand_limbs(rng, 3)
    assert np.array_equal(gpu_lib.mul(z, a), _want(z, a))
    # odd limb offsets on both sides (8-byte aligned buffers)
    buf, out = rand_limbs(rng, 9001), np.zeros(9003, dtype=np.uint64)
    gpu_lib.mul_(out, 1, buf, 3, 5000, buf, 5003, 3998)
    assert np.array_equal(out[1:8999], _want(buf[3:5003].copy(), buf[5003:9001].copy()))


def test_word_batch_equals_fp64_passes(gpu_lib):
    rng = np.random.default_rng(78)
    pairs = [(adversarial(rng, int(m)), None if k % 5 == 0 else adversarial(rng, max(1, int(m * f))))
             for k, (m, f) in enumerate(zip(np.exp(rng.uniform(0, np.log(150000), 120)), rng.uniform(0.01, 1, 120)))]
    got = gpu_lib.mul_batch(pairs)
    old = gpu_lib.get_tuning()
    try:
        t = json.loads(old)
        t["cmax"] = 64  # pass knobs other than the loaded ones: the FP64 passes
        gpu_lib.set_tuning(json.dumps(t))
        assert "k_wtail" not in _kinds(gpu_lib, *pairs[1])
        ref = gpu_lib.mul_batch(pairs)
    finally:
        gpu_lib.set_tuning(old)
    for (a, b), g, r in zip(pairs, got, ref):
        assert np.array_equal(g, r)
        assert np.array_equal(g, _want(a, b))


@pytest.mark.parametrize("k", [1, 31, 32, 33, 64, 65, 96, 97, 128, 192, 256, 257, 384, 512, 513, 768, 769])
def test_power_chains_at_transform_edges(gpu_lib, k):
    # moduli at and around half of each one-CTA length (2k + 1 coefficients:
    # the last one wraps when 2k is the length), extreme limbs, the largest
    # base; 769 limbs: the product batches
    rng = np.random.default_rng(4000 + k)

    def num(x):
        return int.from_bytes(np.ascontiguousarray(x).tobytes(), "little")

    mods, bases, exps = [], [], []
    for style in range(4):
        m = rand_limbs(rng, k)
        if style == 1:
            m[:] = 2**64 - 1
        if style == 2:
            m[:] = 0
            m[-1] = 1 << 13
            m[0] |= np.uint64(3)
        m[0] |= np.uint64(2)
        b = rand_limbs(rng, k) if style != 3 else np.full(k, 2**64 - 1, dtype=np.uint64)
        if style == 1:
            b = m.copy()
            b[0] -= np.uint64(1)
        mods.append(m)
        bases.append(b)
        exps.append(rand_limbs(rng, 1))
    for r, b, e, m in zip(gpu_lib.powermod_batch(bases, exps, mods), bases, exps, mods):
        assert num(r) == pow(num(b), num(e), num(m))


@pytest.mark.parametrize("odd,k", [(1, 22), (3, 21), (1, 23), (3, 22), (1, 24), (3, 23)])
def test_six_prime_shapes(gpu_lib, odd, k):
    # each middle pass (32 to 256 rows) at its exact length; the largest coefficients
    N = odd << k
    rng = np.random.default_rng(N)
    a = rand_limbs(rng, (N + 1) // 2)
    if k == 22:
        a[:] = 2**64 - 1
    assert np.array_equal(gpu_lib.sqr(a), _want(a, None))
    b = rand_limbs(rng, 70001)
    c = rand_limbs(rng, N + 1 - b.size)
    assert np.array_equal(gpu_lib.mul(c, b), _want(c, b))


@pytest.mark.parametrize("m,n", [(200, 150), (1600, 1473), (4864, 4321), (70000, 61000), (250000, 240000)])
def test_host_buffers_pinned_and_pageable(gpu_lib, m, n):
    # one-CTA, direct and staged host products, each operand and the result in
    # pinned or pageable memory
    rng = np.random.default_rng(m)
    a, b = rand_limbs(rng, m), rand_limbs(rng, n)
    want = _want(a, b)

    def buf(x, pinned):
        t = torch.empty(x.size, dtype=torch.int64, pin_memory=pinned)
        v = t.numpy().view(np.uint64)
        v[:] = x
        return t, v

    for mask in range(8):
        (ka, va), (kb, vb), (kr, vr) = (buf(x, bool(mask >> i & 1)) for i, x in enumerate((a, b, np.zeros(m + n, np.uint64))))
        gpu_lib.mul_(vr, 0, va, 0, m, vb, 0, n)
        assert np.array_equal(vr, want)


def test_calls_on_several_streams_share_the_workspace(gpu_lib):
    rng = np.random.default_rng(91)
    streams = [torch.cuda.Stream() for _ in range(3)]
    jobs = []
    torch.cuda.synchronize()
    for k in range(24):
        m, n = int(rng.integers(2000, 60000)), int(rng.integers(500, 30000))
        a, b = rand_limbs(rng, m), rand_limbs(rng, n)
        with torch.cuda.stream(streams[k % 3]):
            da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
            r = torch.zeros(m + n, dtype=torch.uint64, device="cuda")
            gpu_lib.mul_dev(r, da, m, db, n, streams[k % 3])
        jobs.append((a, b, r))
        del da, db  # in flight on the stream
    torch.cuda.synchronize()
    for a, b, r in jobs:
        assert np.array_equal(r.cpu().numpy(), _want(a, b))


@pytest.mark.parametrize("n", [1700, 4096, 9000, 33000, 65536, 66000, 300000])
def test_carries_between_runs(gpu_lib, n):
    # limb sums that overflow and runs of all-ones limbs across many runs, alone
    # (the last pass carries up to 2048 runs itself) and in a batch (a launch does)
    rng = np.random.default_rng(n)
    ones = np.full(n, 2**64 - 1, dtype=np.uint64)
    two = np.zeros(n, dtype=np.uint64)
    two[0] = two[n // 2] = 1
    ends = np.zeros(n, dtype=np.uint64)
    ends[0], ends[-1] = 2**64 - 1, 1 << 63
    third = np.zeros(n // 3 + 1, dtype=np.uint64)
    third[0] = third[-1] = 1
    pairs = [(ones, None), (two, ones), (ends, ones), (ends, None), (ones, third),
             (adversarial(rng, n), adversarial(rng, 2 * n // 3))]
    batch = gpu_lib.mul_batch(pairs)
    for (a, b), g in zip(pairs, batch):
        want = _want(a, b)
        assert np.array_equal(gpu_lib.sqr(a) if b is None else gpu_lib.mul(a, b), want)
        assert np.array_equal(g, want)


@pytest.mark.parametrize("odd,k", [(1, 8), (3, 8), (1, 13), (5, 13), (7, 13), (1, 18), (1, 22), (3, 22)])
def test_limbs_at_packing_edges(gpu_lib, odd, k):
    # upper words at the multiples of p that packing subtracts (p to 3p and the
    # one nearest 2^31, for 30-bit primes of each set), low words that make the
    # reduction's quotient its least and greatest
    n = ((odd << k) + 1) // 2
    rng = np.random.default_rng(n)
    ps = np.array([1073479681, 825753601, 943718401, 415236097, 998244353, 595591169], dtype=np.int64)
    near = np.concatenate([c * ps for c in (1, 2, 3)] + [((1 << 31) + ps // 2) // ps * ps])
    hi = np.unique(np.concatenate([near + d for d in (-1, 0, 1)] + [[0, 1, 2**32 - 1]]))
    lo = np.concatenate([ps, (1 << 32) - ps, [0, 1, 2**31, 2**32 - 1]])
    hi = hi[hi < 2**32].astype(np.uint64)
    a, b = (rng.choice(hi, n) << np.uint64(32) | rng.choice(lo, n).astype(np.uint64) for _ in range(2))
    a[-1] = b[-1] = 2**64 - 1
    assert np.array_equal(gpu_lib.mul(a, b), _want(a, b))
    assert np.array_equal(gpu_lib.sqr(a), _want(a, None))
