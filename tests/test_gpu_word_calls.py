"""Device calls that return before their kernels have run: dependent calls on
one stream, their buffers' lifetimes and their order, against GMP's products."""
import numpy as np
import pytest

import oracle as O
from conftest import rand_limbs

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [40, 177, 700, 1500, 2100, 40000])
@pytest.mark.parametrize("style", ["uniform", "ones"])
def test_dependent_calls_on_one_stream(gpu_lib, n, style):
    # each call reads what the one before wrote, and writes an operand of the
    # calls before it (one-CTA and longer products, before and after one
    # another); all-ones operands: the last pass carries across its runs
    rng = np.random.default_rng(n)
    x = rand_limbs(rng, n) if style == "uniform" else np.full(n, 2**64 - 1, dtype=np.uint64)
    h = n // 2
    dev = {k: torch.zeros(s, dtype=torch.uint64, device="cuda") for k, s in (("x", n), ("p", 2 * n), ("q", 4 * n))}
    dev["x"].copy_(torch.from_numpy(x))
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    rounds = 12
    for _ in range(rounds):
        gpu_lib.sqr_dev(dev["p"], dev["x"], n, st)
        gpu_lib.sqr_dev(dev["q"], dev["p"], 2 * n, st)
        gpu_lib.mul_dev(dev["x"], dev["p"][n:], h, dev["q"][n:], n - h, st)
    torch.cuda.synchronize()
    for _ in range(rounds):
        p = O.gmp_sqr(x)
        q = O.gmp_sqr(p)
        x = O.gmp_mul(p[n: n + h].copy(), q[n: 2 * n - h].copy())
    for k, want in (("p", p), ("q", q), ("x", x)):
        assert np.array_equal(dev[k].cpu().numpy(), want), k


@pytest.mark.parametrize("budget", [320_000_000, 270_000_000])
def test_server_budget_between_the_two_workspaces(gpu_lib, budget):
    # 4.3M output limbs: 302 MB of six-prime residues, 235 MB of FP64 transforms
    n = 2_150_000
    rng = np.random.default_rng(n)
    a, b = rand_limbs(rng, n), rand_limbs(rng, n)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    r = torch.zeros(2 * n, dtype=torch.uint64, device="cuda")
    torch.cuda.synchronize()
    s = gpu_lib.Server(hbm_budget_bytes=budget)
    t = s.submit_dev(r, da, n, db, n, 64 * n, 64 * n)
    s.wait(t)
    s.release(t)
    s.close()
    assert np.array_equal(r.cpu().numpy(), O.gmp_mul(a, b))


@pytest.mark.parametrize("how", ["mul_dev", "mul_batch_dev"])
@pytest.mark.parametrize("n", [500, 500_000])
def test_temporaries_dropped_after_the_call(gpu_lib, how, n):
    # operands allocated under another stream than the call's (the legacy
    # default one), dropped at once, and that stream's next tensors written
    rng = np.random.default_rng(n)
    side = torch.cuda.Stream()
    a, b = rand_limbs(rng, n), rand_limbs(rng, n)
    pa, pb = (torch.from_numpy(x.view(np.int64)).pin_memory() for x in (a, b))
    rs = []
    for _ in range(4):
        with torch.cuda.stream(side):
            da, db = pa.cuda(non_blocking=True), pb.cuda(non_blocking=True)
            r = torch.zeros(2 * n, dtype=torch.int64, device="cuda")
        side.synchronize()
        if how == "mul_dev":
            gpu_lib.mul_dev(r, da, n, db, n)
        else:
            gpu_lib.mul_batch_dev(gpu_lib.make_descs([(r, da, db, n, n, 0, 0)]))
        del da, db
        with torch.cuda.stream(side):
            over = [torch.full((n,), -1, dtype=torch.int64, device="cuda") for _ in range(4)]
        del over
        rs.append(r)
    torch.cuda.synchronize()
    want = O.gmp_mul(a, b)
    for r in rs:
        assert np.array_equal(r.cpu().numpy().view(np.uint64), want)


def _carry_operands(n, rng):
    ones = np.full(n, 2**64 - 1, dtype=np.uint64)
    low = np.zeros(n, dtype=np.uint64)  # the carry starts at the bottom, or in the middle
    low[0] = low[-1] = 1
    mid = low.copy()
    mid[n // 2] = 1
    short = ones[: n // 5 + 1].copy()
    part = ones.copy()  # runs that end inside a tile, at every distance from its start
    part[rng.integers(0, n, n // 40)] = 2**64 - 2
    return [(ones, None), (ones, low), (ones, mid), (ones, short), (part, low), (low, None)]


@pytest.mark.parametrize("n", [1537, 2111, 4096, 8200, 40_000, 131_073, 1 << 21])
def test_long_carries(gpu_lib, n):
    # carries through thousands of tiles (one CTA's fix up to 2048 of them, a
    # launch above, which looks 4096 tiles down at a time), alone and in a batch
    pairs = _carry_operands(n, np.random.default_rng(n))
    want = [O.gmp_sqr(a) if b is None else O.gmp_mul(a, b) for a, b in pairs]
    dev = [tuple(None if x is None else torch.from_numpy(x).cuda() for x in p) for p in pairs]
    for off in (0, 1):  # results at 16 and at 8 bytes
        rs = [torch.zeros(w.size + 2, dtype=torch.uint64, device="cuda")[off:] for w in want]
        torch.cuda.synchronize()
        for r, (a, b) in zip(rs, dev):
            if b is None:
                gpu_lib.sqr_dev(r, a, a.numel())
            else:
                gpu_lib.mul_dev(r, a, a.numel(), b, b.numel())
        torch.cuda.synchronize()
        for k, (r, w) in enumerate(zip(rs, want)):
            got = r.cpu().numpy()
            assert np.array_equal(got[: w.size], w), k
            assert not got[w.size:].any(), k
    if n < 1 << 20:
        for k, (g, w) in enumerate(zip(gpu_lib.mul_batch(pairs), want)):
            assert np.array_equal(g, w), k


@pytest.mark.parametrize("n", [4096, 65_536, 131_072])
def test_carry_runs_are_not_the_products_cost(gpu_lib, n):
    # all-ones operands (every tile passes a carry on) against uniform ones:
    # their carries, tile by tile in one warp, once took eight times the product
    rng = np.random.default_rng(n)
    r = torch.zeros(2 * n, dtype=torch.uint64, device="cuda")
    times = []
    for a in (rand_limbs(rng, n), np.full(n, 2**64 - 1, dtype=np.uint64)):
        da = torch.from_numpy(a).cuda()
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        best = 1e9
        for _ in range(6):
            torch.cuda.synchronize()
            e0.record()
            for _ in range(40):
                gpu_lib.sqr_dev(r, da, n)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1))
        times.append(best)
    assert times[1] < 4 * times[0]


@pytest.mark.parametrize("la,lb,k", [(100, 80, 60), (100, 80, 300), (900, 900, 900), (5000, 4000, 4500), (20_000, 30_000, 20_000),
                                     (60_000, 60_000, 60_000), (60_000, 50_000, 200_000), (600_000, 500_000, 550_000)])
def test_low_products(gpu_lib, la, lb, k):
    # one-CTA, staged, driver-copied and pipelined products, above and below
    # the full product's length
    rng = np.random.default_rng(la + k)
    a, b = rand_limbs(rng, la), rand_limbs(rng, lb)

    def low(full):
        out = np.zeros(k, dtype=np.uint64)
        out[: min(k, full.size)] = full[:k]
        return out

    assert np.array_equal(gpu_lib.mullo(a, b, k), low(O.gmp_mul(a, b)))
    assert np.array_equal(gpu_lib.sqrlo(a, k), low(O.gmp_sqr(a)))
