"""Host side of the benchmark's per-call figures and labels (no GPU)."""
import time

import bench


def test_per_call_latency_includes_the_wait():
    # calls return before their kernels are done: a call's latency ends with the wait
    pending = []

    def call(k):
        pending.append(k)

    def wait():
        time.sleep(0.002 * len(pending))
        pending.clear()

    enqueue, done = bench.per_call_latency(call, wait, 5)
    assert len(enqueue) == len(done) == 5
    assert min(done) >= 2.0 and max(enqueue) < 2.0  # ms


def test_compute_dtype_follows_the_dominant_kernel():
    for k in ("k_wblock", "k_wtail", "k_wsmall"):
        assert bench.compute_dtype(k) == "u32"
    for k in ("k_pwr", "k_fwd", "k_col_tma_fwd", "k_unpack"):
        assert bench.compute_dtype(k) == "f64"
