"""The tree walk (csrc/pc_walk.cuh) against the oracle and the level sweeps, and its FP32 error
bound on the host.

The walk decides leaf or division by the sign of an FP32 time left, settled in FP64 wherever
|time left| is within a bound of its error, so its counts must equal the level sweeps' (which
compare FP64 due times) bit for bit on every input either serves. The host tests restate the
walk's FP32 recurrence with numpy and compare its error with the bound.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def walk_type(built, tmp_path_factory):
    from procell import _lib
    out = str(tmp_path_factory.mktemp("walk") / "libwalk_band.so")
    libdir = os.path.dirname(_lib.LIB_PATH)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(built._cuda_home(), "include"),
                    os.path.join(ROOT, "tests", "walk_band.cpp"), "-o", out, "-L" + libdir, "-lprocell",
                    "-Wl,-rpath," + libdir], check=True)
    ctypes.CDLL(_lib.LIB_PATH, mode=ctypes.RTLD_GLOBAL)
    lib = ctypes.CDLL(out)
    lib.walk_type.restype = ctypes.c_int
    lib.walk_type.argtypes = [ctypes.c_double] * 4 + [ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_uint64)]

    def call(mean, sd, t_max, cum=1.0):
        f, c = (ctypes.c_float * 5)(), ctypes.c_uint64()
        ok = lib.walk_type(mean, sd, t_max, cum, f, ctypes.byref(c))
        return bool(ok), [np.float32(x) for x in f], c.value
    return call


F = np.float32


def fma32(a, b, c):  # a, b, c float32: the product is exact in FP64, one rounding to FP64 and one to FP32
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


@pytest.mark.parametrize("mean,sd,t_max", [(45.0, 13.5, 336.0), (30.0, 0.0, 336.0), (1.0, 3.0, 12.0), (20.0, -6.0, 120.0),
                                           (1e6, 3e5, 336.0), (2.0 ** -20, 2.0 ** -21, 2.0 ** -16), (1e-3, 1e-4, 0.02),
                                           (7.3e8, 2e8, 9e9), (80.0, 20.0, 0.0)])
def test_time_left_stays_within_its_bound(walk_type, mean, sd, t_max):
    ok, (m, s, eps, per_gen, base), _ = walk_type(mean, sd, t_max)
    assert ok
    rng = np.random.default_rng(5)
    n, cap = 200_000, 31
    band = base.astype(np.float64) + cap * per_gen.astype(np.float64)
    z = rng.standard_normal(n).astype(F)
    u_bits = rng.integers(0, 1 << 53, n, dtype=np.uint64)
    sd64 = np.float64(sd)
    keep = sd64 * z + mean > 0
    z, u_bits = z[keep], u_bits[keep]
    tau64 = sd64 * z.astype(np.float64) + mean
    u = (u_bits.astype(np.float64) + 1.0) * 2.0 ** -53
    due = tau64 * u + tau64
    tau = fma32(np.full(z.shape, s), z, np.full(z.shape, m))
    one_u = fma32((u_bits >> np.uint64(29)).astype(np.float64).astype(F), np.full(z.shape, F(2.0 ** -24)), np.ones(z.shape, F))
    rem = (F(t_max) - (tau * one_u).astype(F)).astype(F)
    for _ in range(cap + 1):
        exact = np.float64(t_max) - due
        # a sign taken outside the band is the exact one, and the error itself stays inside it
        # (relative to |rem| for cells far beyond t_max)
        sure = np.abs(rem.astype(np.float64)) > band
        assert np.array_equal((rem < 0)[sure], (exact < 0)[sure])
        assert np.all(np.abs(rem - exact)[exact >= 0] <= band)
        alive = (exact >= 0) & (rem >= 0)
        due, rem = due[alive], rem[alive]
        if not len(due):
            break
        z = rng.standard_normal(len(due)).astype(F)
        tau64 = sd64 * z.astype(np.float64) + mean
        tau = fma32(np.full(z.shape, s), z, np.full(z.shape, m))
        assert np.all(tau64[tau > eps] > 0)  # a timer the walk accepts is positive in FP64
        ok_z = tau64 > 0
        due, rem = due[ok_z] + tau64[ok_z], (rem[ok_z] - tau[ok_z]).astype(F)


def test_ratio_threshold_is_exact(walk_type):
    rng = np.random.default_rng(6)
    for cum in [0.0, 1.0, 0.5, 2.0 ** -53, 1.0 - 2.0 ** -53, 1.0 + 1e-9, -1e-12, 0.1, 1.0 / 3.0] + list(rng.uniform(0, 1, 200)):
        _, _, thr = walk_type(10.0, 1.0, 100.0, float(cum))
        for m in {0, 1, (1 << 53) - 1, max(0, thr - 1), min((1 << 53) - 1, thr)}:
            assert (m < thr) == (m * 2.0 ** -53 < cum), (cum, m)


def test_out_of_range_types_are_refused(walk_type):
    assert not walk_type(1e-30, 1e-31, 10.0)[0]
    assert not walk_type(1e30, 1e29, 10.0)[0]
    assert not walk_type(10.0, 1e30, 10.0)[0]
    assert not walk_type(10.0, 1.0, 1e30)[0]
    assert not walk_type(10.0, 1.0, 1e-30)[0]
    assert walk_type(-1.0, -1.0, 10.0)[0] and walk_type(0.0, 5.0, 10.0)[0]


MANY = [(1.0 / 64, 3.0 + 0.7 * i, 0.5 + 0.1 * i) for i in range(64)]
CASES = {
    "one_cell": ([(3e4, 1)], [(1.0, 10.0, 3.0)], 120.0),
    "warp_edges": ([(900.0, 31), (800.0, 1), (700.0, 32), (600.0, 33), (500.0, 1)], [(0.6, 9.0, 3.0), (0.4, 14.0, 2.0)], 70.0),
    "64_types_one_bin": ([(5e3, 4001)], MANY, 40.0),                    # more classes than window columns
    "64_types_tiny_bins": ([(10.0 + 0.01 * i, 1 + i % 3) for i in range(3000)], MANY, 30.0),
    "no_division": ([(1.5, 1000), (0.2, 50)], [(1.0, 10.0, 2.0)], 500.0),  # phi cap 0: all due cells vanish
    "cap_31": ([(2.0 ** 31.5, 2), (2.0 ** 20, 40)], [(1.0, 2.0, 0.6)], 26.0),
    "cap_32_sweeps": ([(2.0 ** 32.5, 2), (50.0, 40)], [(1.0, 2.0, 0.6)], 24.0),
    "never_leaves": ([(2.0 ** 20.5, 3)], [(1.0, 1.0, 0.1)], 1e6),       # full binary trees: spills, hand-overs
    "fixed_timer": ([(4096.0, 5000)], [(0.5, 12.0, 0.0), (0.5, 0.0, 0.0)], 24.0),
    "zero_mean_at_zero": ([(64.0, 20)], [(1.0, 0.0, 1.0)], 0.0),        # the time left is exactly 0
    "tight_sd": ([(512.0, 4000)], [(1.0, 10.0, 1e-7)], 45.0),
    "mean_beyond_t_max": ([(512.0, 4000)], [(1.0, 1e7, 4e6)], 40.0),
    "heavy_truncation": ([(4096.0, 700)], [(0.5, 1.0, 3.0), (0.5, 2.0, -5.0)], 14.0),
    "out_of_range_sweeps": ([(256.0, 300)], [(1.0, 1e25, 1e24)], 3e25),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
def test_walk_matches_oracle_and_level_sweeps(engine, oracle_lib, name):
    bins, types, t_max = CASES[name]
    p = engine.plan(bins, types, t_max, 1.0, 4242)
    try:
        p.run()
        walk, st = p.raw_counts(), p.stats()
        engine.set_option("sweep_config", 5)  # level sweeps
        p.run()
        level, sl = p.raw_counts(), p.stats()
    finally:
        engine.set_option("sweep_config", 4)
        p.close()
    assert np.array_equal(walk, level)
    for k in ("divisions", "vanished", "uncounted", "max_generation"):
        assert st[k] == sl[k], k
    o = oracle_lib.simulate(bins, types, t_max, 1.0, seed=4242, nthreads=0)
    assert st["divisions"] == o.stats["divisions"] and int(walk.sum()) == o.stats["leaves"]
    assert st["max_generation"] == o.stats["max_gen"]


@pytest.mark.gpu
@pytest.mark.parametrize("lo,hi", [(0, 1), (31, 64), (500, 3333), (4000, 4000), (8998, 9600)])
def test_walk_of_a_root_range(engine, oracle_lib, lo, hi):
    import procell.configs as cfg
    w = cfg.small()
    g = engine.simulate(w.bins, w.types, w.t_max, w.phi, w.seed, root_begin=lo, root_end=min(hi, w.roots))
    o = oracle_lib.simulate(w.bins, w.types, w.t_max, w.phi, seed=w.seed, root_begin=lo, root_end=min(hi, w.roots), nthreads=0)
    assert np.array_equal(g.per_type, o.per_type) and g.stats["divisions"] == o.stats["divisions"]


@pytest.mark.gpu
def test_batch_of_every_case_and_mixed_with_a_deep_one(engine, oracle_lib):
    served = [n for n in sorted(CASES) if not n.endswith("_sweeps") and n != "cap_31"]
    for names in (served, served[:4] + ["cap_32_sweeps"]):
        b = engine.batch([(CASES[n][0], CASES[n][1], CASES[n][2], 1.0, 100 + i) for i, n in enumerate(names)])
        try:
            b.run()
            got = [b.result(i) for i in range(len(names))]
        finally:
            b.close()
        for i, n in enumerate(names):
            o = oracle_lib.simulate(*CASES[n][:3], 1.0, seed=100 + i, nthreads=0)
            assert np.array_equal(got[i].per_type, o.per_type), n


@pytest.mark.gpu
def test_a_walk_without_scratch_goes_to_the_level_sweeps(oracle_lib):
    """Every CUDA call of a context's first run failed in turn: an error status or exact counts,
    and for one of them (the walk's scratch) the level sweeps give them."""
    import procell.configs as cfg
    from procell import Engine, ProcellError
    w = cfg.small()
    o = oracle_lib.simulate(w.bins, w.types, w.t_max, w.phi, seed=w.seed, nthreads=0)
    by_sweeps, n = 0, 1
    while True:
        eng = Engine(0)
        try:
            f0 = eng.get_option("faults_injected")
            eng.set_option("fail_nth_call", n)
            try:
                r = eng.simulate(w.bins, w.types, w.t_max, w.phi, w.seed)
                assert np.array_equal(r.per_type, o.per_type)
                by_sweeps += r.stats["kernel_launches"] > 1
            except ProcellError as e:
                assert e.code in (2, 3), n  # PC_ERR_CUDA, PC_ERR_NOMEM
            if eng.get_option("faults_injected") == f0:  # past the run's last call
                break
        finally:
            eng.close()
        n += 1
    assert n > 5 and by_sweeps == 1


@pytest.mark.gpu
def test_the_memory_budget_bounds_the_scratch(oracle_lib):
    """Setting the budget gives the walk's scratch back; below its size the level sweeps run, and a
    run captured in a graph before is captured again on the new scratch."""
    import procell.configs as cfg
    from procell import Engine
    w = cfg.small()
    o = oracle_lib.simulate(w.bins, w.types, w.t_max, w.phi, seed=w.seed, nthreads=0)
    eng = Engine(0)
    try:
        eng.set_option("driver", 1)
        eng.set_option("graph", 1)
        p = eng.plan(w.bins, w.types, w.t_max, w.phi, w.seed)
        p.run()
        for budget in (1 << 30, 32 << 20, 1 << 30):
            before = eng.get_option("device_allocations")
            eng.set_option("memory_budget_bytes", budget)
            assert eng.get_option("device_allocations") < before
            for _ in range(2):
                p.run()
                assert np.array_equal(p.result().per_type, o.per_type)
            assert (eng.get_option("level_buffers") > 0) == (budget == 32 << 20)
        p.close()
    finally:
        eng.close()


@pytest.mark.gpu
def test_cells_that_are_all_due_at_once_go_to_the_level_sweeps(engine, oracle_lib):
    """Zero-mean types at t_max = 0: a time left of 0 is inside every band, so the walk would settle
    every cell by replaying its lineage."""
    bins, types, t_max = CASES["zero_mean_at_zero"]
    g = engine.simulate(bins, types, t_max, 1.0, 4242)
    o = oracle_lib.simulate(bins, types, t_max, 1.0, seed=4242, nthreads=0)
    assert np.array_equal(g.per_type, o.per_type) and g.stats["divisions"] == o.stats["divisions"]
    assert g.stats["kernel_launches"] > 1  # a walk is one launch


# Timers close to exponential ones (a normal of mean far below its spread, cut at 0): about 5e5
# divisions whose deepest lineages reach the cap of 31, where a node takes all 32 bits.
AT_CAP_31 = ([(2.0 ** 31.5, 2), (2.0 ** 31.2, 1)], [(1.0, 0.25, 10.0)], 120.0)


@pytest.mark.gpu
@pytest.mark.parametrize("driver,graph", [(0, 0), (1, 1)])
def test_lineages_that_reach_the_cap_of_31(engine, oracle_lib, driver, graph):
    o = oracle_lib.simulate(*AT_CAP_31, 1.0, seed=4242, nthreads=0)
    assert o.stats["max_gen"] == 31 and o.stats["vanished"] > 1000
    engine.set_option("driver", driver)
    engine.set_option("graph", graph)
    try:
        g = engine.simulate(*AT_CAP_31, 1.0, 4242)
        b = engine.batch([(*CASES["warp_edges"], 1.0, 7), (*AT_CAP_31, 1.0, 4242), (*CASES["cap_31"], 1.0, 9)])
        b.run()
        in_batch, beside = b.result(1), b.result(2)
        b.close()
    finally:
        engine.set_option("driver", 0)
        engine.set_option("graph", 0)
    assert np.array_equal(g.per_type, o.per_type) and np.array_equal(in_batch.per_type, o.per_type)
    for k in ("divisions", "vanished", "uncounted", "leaves"):
        assert g.stats[k] == o.stats[k], k
    assert g.stats["max_generation"] == 31
    o2 = oracle_lib.simulate(*CASES["cap_31"], 1.0, seed=9, nthreads=0)
    assert np.array_equal(beside.per_type, o2.per_type)


@pytest.mark.gpu
def test_type_choice_of_every_count(engine, oracle_lib):
    """Thresholds are read four at a time and then one by one: 1 to 9 types, and thresholds that do not
    ascend (a negative ratio)."""
    sets = [[(1.0 / n, 8.0 + k, 2.0) for k in range(n)] for n in range(1, 10)]
    sets.append([(0.5, 8.0, 2.0), (0.3, 9.0, 2.0), (0.3, 10.0, 2.0), (0.2, 11.0, 2.0), (-0.3, 12.0, 2.0)])
    bins = [(700.0, 301), (60.0, 77)]
    b = engine.batch([(bins, t, 40.0, 1.0, 60 + i) for i, t in enumerate(sets)])
    b.run()
    for i, t in enumerate(sets):
        o = oracle_lib.simulate(bins, t, 40.0, 1.0, seed=60 + i, nthreads=0)
        assert np.array_equal(b.result(i).per_type, o.per_type), i
        assert np.array_equal(engine.simulate(bins, t, 40.0, 1.0, 60 + i).per_type, o.per_type), i
    b.close()
