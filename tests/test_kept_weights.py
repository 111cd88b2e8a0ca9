"""Weights kept between the passes of a call: one buffer per device for all engines on it, given back with the last."""
import gc
import threading

import numpy as np
import pytest

import oracle as O
from libgwmodel_gb300 import Engine
from libgwmodel_gb300._lib import lib

pytestmark = pytest.mark.gpu


def problem(n, p, seed):
    rng = np.random.default_rng(seed)
    x = np.asfortranarray(np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))]))
    return x, x.sum(1) + rng.normal(0, 0.3, n), np.asfortranarray(rng.uniform(0, 100, (n, 2)))


def fitted(n, p, seed):
    e = Engine(0)
    e.set_data(*problem(n, p, seed))
    return e, e.fit(200, True, O.BISQUARE, False)


def test_one_buffer_for_two_engines_and_none_after_them():
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    gc.collect()  # no engine of an earlier test
    n, p = 20011, 12
    free = lambda: torch.cuda.mem_get_info(0)[0]
    warm = Engine(0)
    start = free()
    a = fitted(n, p, 1)[0]
    one = free()
    b = fitted(n, p, 2)[0]
    two = free()
    assert one - two <= lib().gwgpu_estimate_bytes(n, p, 0, 0, 1)  # without a second 3.2 GB of weights
    del a, b
    weights = 157 * 1251 * 16 * 128 * 8  # row blocks x tiles x points x rows
    assert start - free() >= weights  # an engine is left, and with it the buffer
    del warm
    assert start - free() <= 64 << 20


@pytest.mark.parametrize("n,p", [(3000, 17), (5003, 12)])
def test_engines_in_threads_share_it(n, p):
    """Each engine's fits are those it gives alone, bit for bit, with four at work on streams of their own."""
    want = [fitted(n - k, p, k)[1] for k in range(4)]
    engines = [Engine(0) for _ in range(4)]
    failed = []

    def work(k):
        try:
            for _ in range(6):
                engines[k].set_data(*problem(n - k, p, k))
                got = engines[k].fit(200, True, O.BISQUARE, False)
                assert all(np.array_equal(g, w) for g, w in zip(got, want[k]))
        except Exception as ex:  # noqa: BLE001 (reported by the main thread)
            failed.append((k, repr(ex)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
