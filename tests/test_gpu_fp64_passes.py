"""Products on the FP64 passes, which serve transforms above 2^25 points, pass
knobs other than the loaded ones, products that are short of memory as word
products, and power chains of long moduli: the lengths of every odd multiplier,
large products, batches, and batches that mix them with word products; all
equal to GMP's.  (Integers: no tolerance.)"""
import concurrent.futures as cf
import json
import os

import numpy as np
import pytest

import oracle as O
from conftest import adversarial, rand_limbs
from test_gpu_config_sizes import LANDINGS, _pattern

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _want(a, b):
    return O.gmp_sqr(a) if b is None else O.gmp_mul(a, b)


def _all_want(pairs):
    with cf.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        return list(ex.map(lambda p: _want(*p), pairs))


def _batch(nbgpu, pairs):
    """The pairs as one reusable device batch: kernel kinds, results of a replay."""
    dev = [tuple(None if x is None else torch.from_numpy(x).cuda() for x in p) for p in pairs]
    rs = [torch.zeros(a.size + (a if b is None else b).size, dtype=torch.uint64, device="cuda") for a, b in pairs]
    items = [(r, da, db, a.size, r.numel() - a.size, nbgpu.magnitude_bits(a), nbgpu.magnitude_bits(a if b is None else b))
             for r, (da, db), (a, b) in zip(rs, dev, pairs)]
    torch.cuda.synchronize()
    bt = nbgpu.Batch(nbgpu.make_descs(items))
    kinds = {s["kind"] for s in bt.stats()}
    for _ in range(2):
        bt.run()
    torch.cuda.synchronize()
    bt.close()
    return kinds, [r.cpu().numpy() for r in rs]


@pytest.fixture
def fp64(gpu_lib):
    """The library with a pass split for a length that nothing here uses: its
    other splits are the default ones, and every product runs on the FP64 passes."""
    old = gpu_lib.get_tuning()
    t = json.loads(old)
    t["overrides"] = list(t.get("overrides", [])) + [{"N": 4, "sqr": 0, "pass_ends": [0]}]
    gpu_lib.set_tuning(json.dumps(t))
    yield gpu_lib
    gpu_lib.set_tuning(old)


@pytest.mark.parametrize("n,N", LANDINGS)
def test_odd_lengths(fp64, n, N):
    rng = np.random.default_rng(n)
    a, b = _pattern(rng, n, "uniform"), _pattern(rng, n, "uniform")
    assert fp64.ntt_params(fp64.magnitude_bits(a), fp64.magnitude_bits(b))[1] == N
    want = [_want(a, b), _want(a, None)]
    assert np.array_equal(fp64.mul(a, b), want[0])
    assert np.array_equal(fp64.sqr(a), want[1])
    if n <= 120_000:
        kinds, got = _batch(fp64, [(a, b), (a, None)])
        assert "k_pwr" in kinds and "k_unpack" in kinds and "k_wcarry" in kinds
        assert not kinds & {"k_wsmall", "k_wcol_fwd", "k_wblock", "k_wtail"}
        assert all(np.array_equal(g, w) for g, w in zip(got, want))


@pytest.mark.parametrize("n", [144_000, 1 << 16, 1 << 20])
@pytest.mark.parametrize("kind", ["uniform", "ones", "sparse"])
def test_large(fp64, n, kind):
    rng = np.random.default_rng(n)
    a, b = _pattern(rng, n, kind), _pattern(rng, n, kind)
    assert np.array_equal(fp64.mul(a, b), _want(a, b))
    assert np.array_equal(fp64.sqr(a), _want(a, None))


def test_batch(fp64):
    rng = np.random.default_rng(5)
    m = np.exp(rng.uniform(np.log(152), np.log(65536), 300)).astype(int)
    pairs = [(adversarial(rng, k), None if i % 5 == 0 else adversarial(rng, max(1, int(k * rng.uniform(0.25, 1)))))
             for i, k in enumerate(m)]
    want = _all_want(pairs)
    kinds, got = _batch(fp64, pairs)
    assert not kinds & {"k_wsmall", "k_wcol_fwd", "k_wblock", "k_wtail"}
    assert all(np.array_equal(g, w) for g, w in zip(got, want))
    assert all(np.array_equal(g, w) for g, w in zip(fp64.mul_batch(pairs), want))


@pytest.mark.parametrize("how", ["replayed", "fresh", "host"])
def test_mixed_with_word_products(gpu_lib, how):
    # products of more than 2^25 coefficients and shorter ones in one batch,
    # carries through every tile of both
    rng = np.random.default_rng(25)
    long = np.full((1 << 25) + 77, 2**64 - 1, dtype=np.uint64)
    ones = np.full(70_001, 2**64 - 1, dtype=np.uint64)
    pairs = [(ones, None), (long, ones[:3].copy()), (rand_limbs(rng, 177), rand_limbs(rng, 152)), (ones, ones[:5000].copy()),
             (rand_limbs(rng, (1 << 25) + 1), rand_limbs(rng, 2)), (adversarial(rng, 9000), adversarial(rng, 4001)),
             (rand_limbs(rng, 1_500_000), rand_limbs(rng, 900_000)), (ones[:300].copy(), ones[:200].copy())]
    want = _all_want(pairs)
    if how == "host":
        got = gpu_lib.mul_batch(pairs)
    elif how == "replayed":
        kinds, got = _batch(gpu_lib, pairs)
        assert {"k_unpack", "k_wsmall", "k_wblock", "k_wtail", "k_wcarry"} <= kinds
    else:
        dev = [tuple(None if x is None else torch.from_numpy(x).cuda() for x in p) for p in pairs]
        rs = [torch.zeros(w.size, dtype=torch.uint64, device="cuda") for w in want]
        torch.cuda.synchronize()
        gpu_lib.mul_batch_dev(gpu_lib.make_descs([(r, da, db, a.size, r.numel() - a.size, 0, 0)
                                                  for r, (da, db), (a, b) in zip(rs, dev, pairs)]))
        torch.cuda.synchronize()
        got = [r.cpu().numpy() for r in rs]
    for k, (g, w) in enumerate(zip(got, want)):
        assert np.array_equal(g, w), k


@pytest.mark.parametrize("k", [2, 40, 300, 800, 2100, 6000])
@pytest.mark.parametrize("passes", ["default", "fp64"])
def test_power_chains(gpu_lib, request, k, passes):
    # chains as product batches: long moduli, and a modulus B^(k-1), whose
    # reciprocal has a limb more, among others
    if passes == "fp64":
        request.getfixturevalue("fp64")
    rng = np.random.default_rng(k)
    mods = [rand_limbs(rng, k), np.zeros(k, dtype=np.uint64), np.full(k, 2**64 - 1, dtype=np.uint64)]
    mods[1][-1] = 1
    bases = [rand_limbs(rng, k), np.full(k, 2**64 - 1, dtype=np.uint64), rand_limbs(rng, k)]
    exps = [rand_limbs(rng, 1) >> np.uint64(20) for _ in mods]
    for r, b, e, m in zip(gpu_lib.powermod_batch(bases, exps, mods), bases, exps, mods):
        assert np.array_equal(r, O.gmp_powm(b, e, m))
