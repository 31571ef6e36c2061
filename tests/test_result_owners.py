"""A call that fails may leave arrays in the histograms it was to fill (a host allocation that failed
half way): the Python entry points free them. A stand-in for the library, no GPU."""
import ctypes
import gc

import pytest

import procell
from procell import ProcellError, _lib

BINS, TYPES = [(10.0, 5)], [(1.0, 20.0, 4.0)]


class FailingLibrary:
    """Puts an array into every histogram and fails."""

    def __init__(self):
        self.buffer = ctypes.create_string_buffer(64)
        self.freed = []

    def _fill(self, hs, n):
        for i in range(n):
            hs[i].values = ctypes.cast(self.buffer, type(hs[i].values))
        return 3  # PC_ERR_NOMEM

    def pc_plan_result(self, ctx, plan, hs):
        return self._fill(hs, 1)

    def pc_batch_result(self, ctx, batch, i, hs):
        return self._fill(hs, 1)

    def pc_simulate(self, *args):
        return self._fill(args[-1], 1)

    pc_simulate_shard = pc_simulate

    def pc_simulate_batch(self, ctx, instances, n, hs):
        return self._fill(hs, n)

    def pc_histogram_free(self, h):
        if h._obj.values:
            self.freed.append(ctypes.addressof(h._obj.values.contents))
            h._obj.values = None

    def pc_last_error(self, ctx):
        return b"host allocation"

    def pc_plan_destroy(self, plan):
        pass

    pc_batch_destroy = pc_destroy = pc_plan_destroy


@pytest.mark.parametrize("call", ["simulate", "simulate_shard", "plan_result", "batch_result", "simulate_batch"])
def test_a_failed_call_frees_what_it_left(monkeypatch, call):
    lib = FailingLibrary()
    monkeypatch.setattr(_lib, "_lib", lib)
    eng = procell.Engine.__new__(procell.Engine)
    eng.L, eng.ctx = lib, None
    part = procell.Batch.__new__(procell.Batch) if call == "batch_result" else procell.Plan.__new__(procell.Plan)
    part.engine, part.handle = eng, 1
    run = {"simulate": lambda: eng.simulate(BINS, TYPES, 50.0),
           "simulate_shard": lambda: eng.simulate(BINS, TYPES, 50.0, root_begin=0, root_end=2),
           "plan_result": lambda: part.result(), "batch_result": lambda: part.result(0),
           "simulate_batch": lambda: eng.simulate_batch([(BINS, TYPES, 50.0, None, 0)] * 3)}[call]
    with pytest.raises(ProcellError):
        run()
    gc.collect()
    assert lib.freed == [ctypes.addressof(lib.buffer)] * (3 if call == "simulate_batch" else 1)
