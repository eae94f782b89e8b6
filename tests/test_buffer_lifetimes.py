"""Device calls record their tensors on the stream that uses them (no GPU: the
library and the tensors' device side are stand-ins)."""
import types

import numpy as np
import pytest

import nbgpu

torch = pytest.importorskip("torch")


class DeviceTensor(torch.Tensor):
    """A CPU tensor that says it is on a GPU and notes where it was recorded."""

    recorded: list

    @staticmethod
    def make(n):
        x = torch.zeros(n, dtype=torch.int64).as_subclass(DeviceTensor)
        x.recorded = []
        return x

    is_cuda = property(lambda self: True)
    def get_device(self):
        return 0

    def record_stream(self, s):
        self.recorded.append(s)


@pytest.fixture
def calls(monkeypatch):
    ok = lambda *a: nbgpu.NBG_OK  # noqa: E731
    fake = types.SimpleNamespace(nbg_mul_dev=ok, nbg_sqr_dev=ok, nbg_mul_batch_dev=ok)
    monkeypatch.setattr(nbgpu, "lib", lambda: fake)
    monkeypatch.setattr(torch.cuda, "default_stream", lambda device=None: "default")
    monkeypatch.setattr(torch.cuda, "ExternalStream", lambda p, device=None: f"external {p}")
    monkeypatch.setattr(nbgpu, "_default_streams", {}, raising=False)


class Stream:
    cuda_stream = 0x70


@pytest.mark.parametrize("stream,where", [(None, "default"), (0, "default"), (Stream, None), (0x30, "external 48")])
def test_calls_record_their_tensors(calls, stream, where):
    s = Stream() if stream is Stream else stream
    where = s if where is None else where
    r, a, b = (DeviceTensor.make(n) for n in (8, 4, 4))
    nbgpu.mul_dev(r, a, 4, b, 4, s)
    assert [x.recorded for x in (r, a, b)] == [[where]] * 3
    nbgpu.sqr_dev(r, a, 4, s)
    assert (r.recorded, a.recorded) == ([where] * 2, [where] * 2)
    # descriptors hold addresses only: the array keeps the tensors
    nbgpu.mul_batch_dev(nbgpu.make_descs([(r, a, None, 4, 4, 0, 0)]), s)
    assert (r.recorded, a.recorded, b.recorded) == ([where] * 3, [where] * 3, [where])
    d = nbgpu.make_descs([(DeviceTensor.make(8), DeviceTensor.make(4), DeviceTensor.make(4), 4, 4, 0, 0)])
    kept = list(d.tensors)
    nbgpu.mul_batch_dev(d, s)
    assert [x.recorded for x in kept] == [[where]] * 3
    # raw addresses are the caller's
    nbgpu.mul_dev(1 << 20, 2 << 20, 4, 3 << 20, 4, s)
    nbgpu.mul_batch_dev(nbgpu.make_descs([(1 << 20, 2 << 20, None, 4, 4, 0, 0)]), s)


def test_results_of_a_batch_do_not_hold_each_other(monkeypatch):
    # a kept result keeps at most the few MB it was allocated with
    fake = types.SimpleNamespace(nbg_mul_batch=lambda *a: nbgpu.NBG_OK)
    monkeypatch.setattr(nbgpu, "lib", lambda: fake)
    sizes = [1, 100, 200_000, 3000, 131_072, 70_000, 1_000_000] * 5 + [2000] * 1000
    pairs = [(np.ones(n, np.uint64), None if n % 3 else np.ones(n, np.uint64)) for n in sizes]
    res = nbgpu.mul_batch(pairs)
    assert [r.size for r in res] == [2 * n for n in sizes]
    spans = []
    for r in res:
        base = r if r.base is None else r.base
        assert base.nbytes <= max(8 << 20, r.nbytes)
        if r.nbytes >= 4 << 20:
            assert r.base is None
        spans.append((r.ctypes.data, r.ctypes.data + r.nbytes))
    spans.sort()
    assert all(x[1] <= y[0] for x, y in zip(spans, spans[1:]))
    assert nbgpu.mul_batch(pairs[:1])[0].size == 2
