"""sampo_step_noalloc at the smallest pools, at the edges of tiles and on both
sides of the largest pool that takes the one-launch step, against sampo_step
with three kernels: the row, the next ranges and counters and every field of
every live slot are identical."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 0, 0, 0), (0, 0, 0, 1), (127, 128, 129, 257), (2003, 1499, 501, 1001), "limit", "past"])
def test_step_noalloc_sizes(gpu_ready, sizes):
    torch = pytest.importorskip("torch")
    from sampo_gb300 import _lib, inputs
    from sampo_gb300.population import make_pool
    from sampo_gb300.sim import Simulation, pop_from_ranges, seed_stream
    from tests.test_zz_no_alloc import _device_pool, _download, _upload
    lib = _lib.load()
    cc, T = 4000.0, np.array([29.0], np.float32)
    env = np.zeros(1, dtype=inputs.ENV_DTYPE)
    env["bloodmealSuccess"] = 0.5
    env["carryingCapacity"] = cc
    env["oviTrapValue"] = 0.05
    _, seeds = seed_stream(3, 1)
    cap = 1 << 16
    if isinstance(sizes, str):  # the last pool of one 1024-slot tile per CTA, and the first larger one
        with Simulation(capacity=1024, carrying_capacity=cc, max_steps=2) as sim:
            slots = sim.small_step_info()["grid"] * 1024
        end = int(make_pool((0, 90000, 20000, 50000), T[0], seed=7)[0][7][1])
        sizes = (slots - end + (0 if sizes == "limit" else 128), 90000, 20000, 50000)
        cap = 1 << 20
    ranges, arrays = make_pool(sizes, T[0], seed=7)
    for hour in (10, 19):
        with Simulation(capacity=cap, carrying_capacity=cc, max_steps=2) as sim:
            sim.set_inputs(T, env)
            sim.set_small_step(0)
            sim.load_pool(ranges, arrays)
            want = sim.step(env[0], T[0], hour, seeds[0])
            after, (pop, pool) = sim.current_row(), sim.read_pool()
        tin, din = _device_pool(torch, cap)
        tout, dout = _device_pool(torch, cap)
        _upload(torch, tin, ranges, arrays)
        torch.cuda.synchronize()
        p, e = pop_from_ranges(ranges), _lib.Environment(*[float(env[0][k]) for k in inputs.ENV_DTYPE.names])
        s = np.ascontiguousarray(seeds[0], dtype=np.uint32)
        row, out, bnc = _lib.StatsRow(), _lib.Population(), _lib.BitesCycles()
        assert lib.sampo_step_noalloc(C.byref(din), cap, C.byref(dout), cap, C.byref(p), C.byref(e), float(T[0]), hour,
                                      s.ctypes.data, cc, C.byref(row), C.byref(out), C.byref(bnc), 0, None) == 0
        assert bytes(row) == want.tobytes()
        assert bytes(out) + bytes(bnc) == after.tobytes()
        got = _download(tout, int(out.r[7].end))
        for k in range(8):
            a, b = (int(x) for x in pop["ranges"][k])
            for name in got:
                assert got[name][a:b].tobytes() == pool[name][a:b].tobytes(), f"range {k} field {name}"
