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


KEPT = r'''
import gc, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import test_results as T
from procell import Engine

def kept():
    e = Engine(0)
    n = e.get_option("result_memory")
    e.close()
    return n

two = [Engine(0), Engine(0)]
small = [two[0].simulate(*T.wide_input(s, bins=2000)) for s in range(3)]  # pages, below the pinned threshold
large = [two[1].simulate(*T.wide_input(s)) for s in range(5)]             # pinned blocks and pages
want = [r.per_type.copy() for r in large]
del small
two[0].close()
assert two[1].get_option("result_memory") > 0
two[1].close()
held = kept()
assert held > 0, held  # the pinned blocks of the results still held
for r, w in zip(large, want):
    assert np.array_equal(r.per_type, w)
del r, large
gc.collect()
assert kept() == 0, kept()
e = Engine(0)  # and again from nothing
r = e.simulate(*T.wide_input(3))
assert np.array_equal(r.per_type, want[3])
e.close()
print("kept ok")
'''


def test_kept_memory_goes_back_with_the_last_context(built):
    """In a process of its own, where no other context is alive."""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    pkg = os.path.join(os.path.dirname(here), "cuda-pro-cell_gb300")
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([pkg, os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", KEPT, here], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.stdout[-1000:], r.stderr[-3000:])
    assert "kept ok" in r.stdout
