"""Performance cases of the big-integer product engine.

Each case is one call pattern of a program that uses `nbgpu`: single products
and squares on device buffers from the NTT admission size (152 limbs) to 2^24
limbs, an unbalanced product, the host-buffer drop-in call, replayed and
one-shot batches of products of mixed sizes, host-buffer batches, Barrett
power chains, and the continuous-batching server.  Limbs are uniform random
64-bit words (or 1% nonzero for the sparse pattern) with a nonzero top limb;
limb buffers on the device are int64 tensors holding the words' bit patterns.
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "nativebigint.jl_b200"))
import nbgpu  # noqa: E402


def listed() -> list[dict]:
    return [
        # the smallest product the reference sends to the NTT: call latency
        dict(name="mul_177x152", kind="mul", m=177, n=152, pattern="uniform"),
        # ordinary operand of a library that squares (roots, powers): one call
        dict(name="sqr_4096", kind="sqr", m=4096, pattern="uniform"),
        # the benchmark's largest mixed-batch operand, ragged, called alone
        dict(name="mul_65536x65521", kind="mul", m=65536, n=65521, pattern="uniform"),
        # million-limb products of binary-splitting trees: the operands' ratio is not 1
        dict(name="mul_1048576x774143", kind="mul", m=1048576, n=774143, pattern="uniform"),
        # the largest single-product configuration of the benchmark
        dict(name="sqr_16777216", kind="sqr", m=1 << 24, pattern="uniform"),
        # unbalanced: a long operand times a short one (one step of a division)
        dict(name="mul_1000003x1021", kind="mul", m=1000003, n=1021, pattern="uniform"),
        # the drop-in call from host memory (what the Julia binding makes)
        dict(name="host_mul_4864x4321", kind="host_mul", m=4864, n=4321, pattern="uniform"),
        # the headline workload: 10,000 independent products, replayed on resident operands
        dict(name="batch_10000", kind="batch", count=10000, lo=152, hi=65536, sizes=1, pattern="uniform"),
        # a fresh batch of device products each call (one tree level of a product tree)
        dict(name="batch_once_256", kind="batch_once", count=256, lo=152, hi=65536, sizes=2, pattern="uniform"),
        # a batch from and to host memory, copies included
        dict(name="host_batch_60", kind="host_batch", count=60, lo=152, hi=65536, sizes=3, pattern="uniform"),
        # modular powers for 16384-bit moduli (primality tests), 1024-bit exponents
        dict(name="powmod_64x256", kind="powmod", count=64, k=256, le=16, pattern="uniform"),
        # a serving burst: requests of mixed sizes submitted together, all awaited
        dict(name="server_256", kind="server", count=256, lo=152, hi=131072, sizes=4, pattern="uniform"),
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["mul", "mul", "mul", "sqr", "sqr", "skew", "host_mul", "batch", "batch", "batch_once",
                       "host_batch", "powmod", "server"])
    pattern = "sparse" if rng.random() < 0.15 else "uniform"
    if kind == "mul":
        m = _log(rng, 152, 1 << 23)
        return dict(kind="mul", m=m, n=max(64, round(m * rng.uniform(0.25, 1.0))), pattern=pattern)
    if kind == "sqr":
        return dict(kind="sqr", m=_log(rng, 160, 1 << 24), pattern=pattern)
    if kind == "skew":
        return dict(kind="mul", m=_log(rng, 20000, 2000000), n=_log(rng, 64, 5000), pattern=pattern)
    if kind == "host_mul":
        m = _log(rng, 152, 200000)
        return dict(kind="host_mul", m=m, n=max(64, round(m * rng.uniform(0.25, 1.0))), pattern=pattern)
    if kind == "powmod":
        return dict(kind="powmod", count=_log(rng, 8, 64), k=_log(rng, 64, 400), le=rng.randint(2, 16),
                    pattern="uniform")
    hi = _log(rng, 1500, 65536)
    count = {"batch": (64, 8000), "batch_once": (16, 512), "host_batch": (8, 60), "server": (32, 256)}[kind]
    return dict(kind=kind, count=_log(rng, *count), lo=152, hi=hi, sizes=rng.randrange(1 << 30), pattern=pattern)


def _sizes(case: dict) -> list[tuple[int, int, bool]]:
    """(m, n, square) per product: m log-uniform in [lo, hi], n/m uniform in
    [0.25, 1], one in five a square (the benchmark's mix)."""
    rng = np.random.Generator(np.random.PCG64(case["sizes"]))
    c = case["count"]
    m = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), c)).astype(np.int64)
    n = np.maximum(1, np.round(m * rng.uniform(0.25, 1.0, c)).astype(np.int64))
    sq = rng.random(c) < 0.2
    return [(int(a), int(a if s else b), bool(s)) for a, b, s in zip(m, n, sq)]


def _shapes(case: dict) -> list[tuple[int, int, bool]]:
    if case["kind"] in ("mul", "host_mul"):
        return [(case["m"], case["n"], False)]
    if case["kind"] == "sqr":
        return [(case["m"], case["m"], True)]
    return _sizes(case)


def _limbs(total: int, tops: np.ndarray, pattern: str, seed: int) -> torch.Tensor:
    """`total` random limbs on the GPU, those at `tops` nonzero."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (total,), dtype=torch.int64, device="cuda", generator=g)
    if pattern == "sparse":
        x *= (torch.rand(total, device="cuda", generator=g) < 0.01).to(torch.int64)
    t = torch.from_numpy(tops).cuda()
    v = x[t]
    x[t] = torch.where(v == 0, torch.ones_like(v), v)
    return x


class _State:
    """Operand and result buffers of a case, plus the handle its program keeps."""


def prepare(case: dict, seed: int) -> _State:
    st = _State()
    st.kind = case["kind"]
    if st.kind == "powmod":
        st.args = _powmod_inputs(case, seed)
        return st
    shapes = _shapes(case)
    st.shapes = shapes
    sizes = np.array([[m, 0 if sq else n] for m, n, sq in shapes], dtype=np.int64).reshape(-1)
    ends = np.cumsum(sizes)
    offs = ends - sizes
    st.x = _limbs(int(ends[-1]), ends[sizes > 0] - 1, case["pattern"], seed)
    if st.kind in ("host_mul", "host_batch"):
        h = st.x.cpu().numpy().view(np.uint64)
        st.pairs = [(h[offs[2 * i]: ends[2 * i]], None if sq else h[offs[2 * i + 1]: ends[2 * i + 1]])
                    for i, (m, n, sq) in enumerate(shapes)]
        del st.x
        return st
    a = [st.x[offs[2 * i]: ends[2 * i]] for i in range(len(shapes))]
    b = [None if sq else st.x[offs[2 * i + 1]: ends[2 * i + 1]] for i, (m, n, sq) in enumerate(shapes)]
    rlen = np.array([m + n for m, n, _ in shapes], dtype=np.int64)
    rend = np.cumsum(rlen)
    st.r = torch.zeros(int(rend[-1]), dtype=torch.int64, device="cuda")
    st.a, st.b = a, b
    st.outs = [st.r[e - ln: e] for e, ln in zip(rend, rlen)]
    if st.kind in ("mul", "sqr"):
        return st
    # magnitude bits of every operand, which a batching program knows
    tops = st.x[torch.from_numpy(np.maximum(ends, 1) - 1).cuda()].cpu().numpy().view(np.uint64)
    bits = [64 * (int(s) - 1) + int(t).bit_length() if s else 0 for s, t in zip(sizes, tops)]
    xp, rp = st.x.data_ptr(), st.r.data_ptr()
    items = [(rp + 8 * int(rend[i] - rlen[i]), xp + 8 * int(offs[2 * i]), None if sq else xp + 8 * int(offs[2 * i + 1]),
              m, n, bits[2 * i], bits[2 * i] if sq else bits[2 * i + 1]) for i, (m, n, sq) in enumerate(shapes)]
    if st.kind == "server":
        st.items = items
        st.server = nbgpu.Server(hbm_budget_bytes=4 << 30)
        return st
    st.descs = nbgpu.make_descs(items)
    if st.kind == "batch":
        torch.cuda.synchronize()
        st.batch = nbgpu.Batch(st.descs)
    return st


def _powmod_inputs(case: dict, seed: int):
    rng = np.random.Generator(np.random.PCG64(seed))
    c, k, le = case["count"], case["k"], case["le"]

    def words(n):
        return rng.integers(0, 2**64, n, dtype=np.uint64)

    mods, bases, exps = [words(k) for _ in range(c)], [words(k) for _ in range(c)], [words(le) for _ in range(c)]
    for m, e in zip(mods, exps):
        m[0] |= np.uint64(1)
        m[-1] |= np.uint64(1 << 63)
        e[-1] |= np.uint64(1 << 63)
    return bases, exps, mods


def run(state: _State):
    k = state.kind
    if k == "mul":
        (m, n, _), = state.shapes
        nbgpu.mul_dev(state.r, state.a[0], m, state.b[0], n)
        return state.r
    if k == "sqr":
        (m, _, _), = state.shapes
        nbgpu.sqr_dev(state.r, state.a[0], m)
        return state.r
    if k == "host_mul":
        (a, b), = state.pairs
        return nbgpu.mul(a, b)
    if k == "host_batch":
        return nbgpu.mul_batch(state.pairs)
    if k == "batch":
        state.batch.run()
        return state.r
    if k == "batch_once":
        nbgpu.mul_batch_dev(state.descs)
        return state.r
    if k == "powmod":
        return nbgpu.powermod_batch(*state.args)
    tickets = [state.server.submit_dev(r, a, m, b, n, ba, bb) for r, a, b, m, n, ba, bb in state.items]
    for t in tickets:
        state.server.wait(t)
    for t in tickets:
        state.server.release(t)
    return state.r


def _transform_ops(limbs: int, transforms: int) -> float:
    # a product of `limbs` output limbs through transforms over word-size
    # primes: about 5 points per limb, 3 operations per point and level
    return 15.0 * limbs * max(1.0, math.log2(limbs)) * transforms


def work(case: dict) -> dict:
    if case["kind"] == "powmod":
        c, k, le = case["count"], case["k"], case["le"]
        steps = 64 * le * 1.2
        return {"bytes": 8.0 * c * (3 * k + le), "flops": c * steps * 3 * _transform_ops(2 * k, 3)}
    by = fl = 0.0
    for m, n, sq in _shapes(case):
        by += 8.0 * ((m if sq else m + n) + m + n)
        fl += _transform_ops(m + n, 2 if sq else 3)
    return {"bytes": by, "flops": fl}


def _int(x: np.ndarray) -> int:
    return int.from_bytes(np.ascontiguousarray(x).tobytes(), "little")


def _words(v: int, n: int) -> np.ndarray:
    return np.frombuffer(v.to_bytes(8 * n, "little"), dtype="<u8").astype(np.uint64)


def exact(case: dict, seed: int):
    """The results by Python's own integers, where those take a few seconds at most."""
    if case["kind"] == "powmod":
        bases, exps, mods = _powmod_inputs(case, seed)
        if case["count"] * case["le"] * case["k"] ** 2 > 2e7:
            return None
        return [_words(pow(_int(b), _int(e), _int(m)), m.size) for b, e, m in zip(bases, exps, mods)]
    shapes = _shapes(case)
    if sum(float(m) * float(n) ** 0.585 for m, n, _ in shapes) > 1e9:
        return None
    sizes = np.array([[m, 0 if sq else n] for m, n, sq in shapes], dtype=np.int64).reshape(-1)
    ends = np.cumsum(sizes)
    offs = ends - sizes
    h = _limbs(int(ends[-1]), ends[sizes > 0] - 1, case["pattern"], seed).cpu().numpy()
    out = []
    for i, (m, n, sq) in enumerate(shapes):
        a = _int(h[offs[2 * i]: ends[2 * i]])
        b = a if sq else _int(h[offs[2 * i + 1]: ends[2 * i + 1]])
        out.append(_words(a * b, m + n))
    if case["kind"] == "host_mul":
        return out[0]
    if case["kind"] == "host_batch":
        return out
    return torch.from_numpy(np.concatenate(out).view(np.int64))
