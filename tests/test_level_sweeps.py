"""The level sweeps of the default configuration, which the tree walk leaves only the runs that it
does not serve: a cap on the size of a sweep (max_slice_cells, far above any level here) sends every
run to them. Counts against the oracle, every failing CUDA call, and the bounds-checked build, whose
copy here also gives the walk a region of 64 cells per warp: runs with deep stacks overflow it, set
their error bit and are run again by the sweeps."""
import os
import subprocess
import sys

import numpy as np
import pytest

import procell.configs as cfg
from test_faults import sweep_faults

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cuda-pro-cell_gb300")
DRIVERS = [(0, 0), (1, 0), (1, 1)]  # (driver, graph)
NO_WALK = float(1 << 40)


@pytest.fixture
def sweeps(built):
    """An engine of its own (its level buffers show that the sweeps ran)."""
    from procell import Engine
    eng = Engine(0)
    eng.set_option("max_slice_cells", NO_WALK)
    yield eng
    eng.close()


@pytest.mark.parametrize("driver,graph", DRIVERS)
@pytest.mark.parametrize("name", ["small", "medium"])
def test_default_configuration_against_the_oracle(sweeps, oracle_lib, name, driver, graph):
    w = cfg.by_name(name)
    o = oracle_lib.simulate(w.bins, w.types, w.t_max, w.phi, seed=w.seed, nthreads=0)
    sweeps.set_option("driver", driver)
    sweeps.set_option("graph", graph)
    g = sweeps.simulate(w.bins, w.types, w.t_max, w.phi, w.seed)
    assert sweeps.get_option("level_buffers") > 0
    assert np.array_equal(g.per_type, o.per_type) and g.stats["divisions"] == o.stats["divisions"]
    b = sweeps.batch([(w.bins, w.types[::-1], w.t_max, w.phi, w.seed), (w.bins, w.types, w.t_max, w.phi, w.seed)])
    b.run()
    assert np.array_equal(b.result(1).per_type, o.per_type)
    b.close()


@pytest.mark.parametrize("driver,graph", DRIVERS)
@pytest.mark.parametrize("batched", [False, True])
def test_every_failing_call_is_reported(sweeps, oracle_lib, batched, driver, graph):
    w = cfg.small()
    o = oracle_lib.simulate(w.bins, w.types, w.t_max, w.phi, seed=w.seed, nthreads=0)
    sweeps.set_option("driver", driver)
    sweeps.set_option("graph", graph)

    def run():
        if not batched:
            return sweeps.simulate(w.bins, w.types, w.t_max, w.phi, w.seed)
        b = sweeps.batch([(w.bins, w.types, w.t_max, w.phi, w.seed)])
        try:
            b.run()
            return b.result(0)
        finally:
            b.close()

    def check(g):
        assert np.array_equal(g.per_type, o.per_type)

    assert sweep_faults(sweeps, run, check) >= 8
    assert sweeps.get_option("level_buffers") > 0


CHECKED = r'''
import numpy as np
import oracle
import procell.configs as cfg
from procell import Engine, _lib
assert _lib.LIB_PATH.endswith("limits/libprocell.so"), _lib.LIB_PATH
DEEP = [("bright", [(2.0 ** 20.5, 3)], [(1.0, 1.0, 0.1)], 1e6), ("spread", [(2.0 ** 31.5, 2)], [(1.0, 0.25, 10.0)], 120.0)]
for name, bins, types, t_max in DEEP:  # stacks beyond the walk's region
    o = oracle.simulate(bins, types, t_max, 1.0, seed=11, nthreads=0)
    for batched in (False, True):
        eng = Engine(0)
        if batched:
            b = eng.batch([([(300.0, 40)], types, 4.0, 1.0, 5), (bins, types, t_max, 1.0, 11)])
            b.run()
            g, divisions = b.result(1), None
            b.close()
        else:
            g = eng.simulate(bins, types, t_max, 1.0, 11)
            assert g.stats["divisions"] == o.stats["divisions"]
        assert eng.get_option("level_buffers") > 0, (name, batched)  # the sweeps ran it again
        assert np.array_equal(g.per_type, o.per_type), (name, batched)
        eng.close()
eng = Engine(0)
eng.set_option("max_slice_cells", 2.0 ** 40)
w0, deep = cfg.small(), ([(2.0 ** 33.5, 2), (50.0, 40)], [(1.0, 2.0, 0.6)], 24.0, 1.0, 3)  # narrow and wide keys
for bins, types, t_max, phi, seed in ((w0.bins, w0.types, w0.t_max, w0.phi, w0.seed), deep):
    o = oracle.simulate(bins, types, t_max, phi, seed=seed, nthreads=0)
    for driver, graph in ((0, 0), (1, 0), (1, 1)):
        eng.set_option("driver", driver)
        eng.set_option("graph", graph)
        g = eng.simulate(bins, types, t_max, phi, seed)  # raises on a failed check
        assert np.array_equal(g.per_type, o.per_type)
        b = eng.batch([(bins, types, t_max, phi, seed), (bins, types, t_max, phi, seed + 1)])
        b.run()
        assert np.array_equal(b.result(0).per_type, o.per_type)
        b.close()
assert eng.get_option("level_buffers") > 0
eng.close()
print("limits ok")
'''


def test_checked_sweeps_and_a_walk_that_outgrows_its_region(built, oracle_lib):
    lib = built.build(out=os.path.join(PKG, "build_checked", "limits"),
                      defines=["PC_CHECKED=1", "PC_WALK_REGION_CELLS=64"])
    env = dict(os.environ, PROCELL_LIB=lib,
               PYTHONPATH=os.pathsep.join([PKG, os.path.join(ROOT, "oracle"), os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", CHECKED], env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, (r.stdout[-2000:], r.stderr[-3000:])
    assert "limits ok" in r.stdout
