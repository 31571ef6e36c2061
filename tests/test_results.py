"""Result arrays are the library's own memory, handed out without a copy (pinned blocks and
kept pages for large ones): results that are held must not change when later ones are made,
memory comes back when the last array on it is gone, and worker threads serve callers that
overlap."""
import gc
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def wide_input(seed, bins=6000):  # about 40,000 values x (1 + 3) counts: above the pinned threshold
    rng = np.random.default_rng(seed)
    v = np.exp(rng.uniform(0, np.log(1e4), bins))
    return ((v, np.full(bins, 2, np.uint64)), [(0.5, 40.0, 8.0), (0.3, 60.0, 9.0), (0.2, -1.0, -1.0)], 200.0, 1.0, seed)


def test_held_results_stay(engine):
    inputs = [wide_input(s) for s in range(7)]
    held = [engine.simulate(*x) for x in inputs]  # more than there are pinned blocks
    copies = [(r.values.copy(), r.totals.copy(), r.per_type.copy()) for r in held]
    part = held[2].per_type[5:9]  # a view alone keeps its memory
    want = part.copy()
    del held[2]
    gc.collect()
    for x, c in zip(inputs, copies):
        r = engine.simulate(*x)
        assert np.array_equal(r.values, c[0]) and np.array_equal(r.totals, c[1]) and np.array_equal(r.per_type, c[2])
        r.totals[:] = 7  # arrays are writable and the caller's own
    assert np.array_equal(part, want)
    for r, c in zip(held, copies[:2] + copies[3:]):
        assert np.array_equal(r.totals, c[1]) and np.array_equal(r.per_type, c[2])


def test_batches_from_overlapping_threads(built):
    from procell import Engine
    instances = [wide_input(20 + i, bins=300) for i in range(24)]
    errors, got = [], [None, None]

    def work(k):
        try:
            e = Engine(0)
            for _ in range(4):
                got[k] = e.simulate_batch(instances)
            e.close()
        except Exception as x:  # noqa: BLE001
            errors.append(x)
    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors
    for a, b in zip(*got):
        assert np.array_equal(a.values, b.values) and np.array_equal(a.per_type, b.per_type)
