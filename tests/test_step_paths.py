"""The routes a step can take, at the sizes where they can go wrong: the
three-kernel day against the CPU oracle at the edges of chunks, rows and
spans, on pools whose records follow from their state (read and written by
their own columns only) and on pools with free records (moved whole); and the
one-launch day of a species compiled at run time against its three-kernel
day. All results are whole records and counts: equal, bit for bit."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HOT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "species", "hot_species.h")


def _workload(sizes, n, cc, seed):
    from sampo_gb300 import inputs
    from sampo_gb300.population import make_pool
    from sampo_gb300.sim import seed_stream
    T = np.linspace(24.0, 31.0, n).astype(np.float32)
    env = np.zeros(n, dtype=inputs.ENV_DTYPE)
    env["bloodmealSuccess"] = 0.5
    env["carryingCapacity"] = cc
    for name in ("ITNValue", "IRSValue", "larvacideValue", "oviTrapValue"):
        env[name][n // 2:] = 0.05
    ranges, arrays = make_pool(sizes, T[0], seed=seed)
    return ranges, arrays, T, env, seed_stream(seed, n)[1]


def _same_pools(ranges, a, b):
    for k in range(8):
        s, e = int(ranges[k][0]), int(ranges[k][1])
        for name in a:
            assert a[name][s:e].tobytes() == b[name][s:e].tobytes(), f"range {k} field {name}"


@pytest.mark.parametrize("free", [False, True])
@pytest.mark.parametrize("sizes", [(1, 0, 0, 0), (0, 1, 1, 1), (31, 32, 33, 65), (127, 128, 129, 257), (1025, 4097, 640, 2053),
                                   (66000, 50001, 9000, 16001)])
def test_three_kernel_day_matches_oracle(gpu_ready, oracle_mod, sizes, free):
    from oracle import OracleSim
    from sampo_gb300.sim import Simulation
    n, cc, cap = 30, 30000.0, 1 << 20   # a day that decides ahead, then six single hours
    ranges, arrays, T, env, seeds = _workload(sizes, n, cc, seed=sum(sizes))
    if free:  # fields that a fresh egg or larva does not have
        for k in (0, 1):
            s, e = int(ranges[k][0]), int(ranges[k][1])
            arrays["numEggBatches"][s:e:3] = 5
            arrays["hoursInState"][s:e:2] += np.float32(0.25)
    orc = OracleSim(cap)
    orc.load_pool(ranges, arrays)
    with Simulation(capacity=cap, carrying_capacity=cc, max_steps=n + 1) as sim:
        sim.set_inputs(T, env)
        sim.set_seeds(0, seeds)
        sim.set_small_step(0)
        sim.load_pool(ranges, arrays)
        rows = sim.run(n)
        assert sim.device_status() & 0xFF == 0
        pop, pool = sim.read_pool()
    for i in range(n):
        assert rows[i].tobytes() == orc.step(env[i], T[i], i % 24, seeds[i]).tobytes(), f"step {i}"
    ro, ao = orc.read_pool()
    assert np.array_equal(np.asarray(pop["ranges"], np.int64), np.asarray(ro, np.int64))
    _same_pools(ro, pool, ao)


@pytest.mark.parametrize("sizes", [(1, 0, 0, 0), (255, 257, 129, 300), (40000, 30000, 9000, 20000)])
def test_species_one_launch_day(gpu_ready, sizes):
    from sampo_gb300.sim import Simulation
    from sampo_gb300.species import Species
    n, cc = 72, 40000.0
    ranges, arrays, T, env, seeds = _workload(sizes, n, cc, seed=5)
    runs = {}
    with Species(HOT) as sp:
        for key, tiles, items in (("three kernels", 0, 0), ("default", None, 0), ("1", None, 1), ("2", None, 2), ("4", None, 4)):
            with Simulation(capacity=1 << 20, carrying_capacity=cc, max_steps=n + 1) as sim:
                sim.set_species(sp)
                sim.set_inputs(T, env)
                sim.set_seeds(0, seeds)
                sim.set_small_step(tiles)
                sim.set_small_step_items(items)
                sim.load_pool(ranges, arrays)
                rows = sim.run(n)
                assert sim.device_status() & 0xFF == 0
                assert sim.small_step_info()["days_one_launch"] == (0 if tiles == 0 else n // 24)
                runs[key] = rows, *sim.read_pool()
    rows, pop, pool = runs.pop("three kernels")
    for key, (r, p, a) in runs.items():
        assert r.tobytes() == rows.tobytes(), key
        assert np.array_equal(p["ranges"], pop["ranges"]), key
        _same_pools(pop["ranges"], a, pool)


@pytest.mark.parametrize("sizes", [(1, 0, 0, 0), (255, 1, 128, 130), (257, 256, 255, 1025), (60000, 40001, 9000, 20000)])
def test_single_hours_match_oracle(gpu_ready, oracle_mod, sizes):
    """sampo_step, one launch an hour and three, with a pool read between."""
    from oracle import OracleSim
    from sampo_gb300.sim import Simulation
    n, cc, cap = 6, 30000.0, 1 << 20
    ranges, arrays, T, env, seeds = _workload(sizes, n, cc, seed=9)
    for tiles in (None, 0):
        orc = OracleSim(cap)
        orc.load_pool(ranges, arrays)
        with Simulation(capacity=cap, carrying_capacity=cc, max_steps=n + 1) as sim:
            sim.set_inputs(T, env)
            sim.set_small_step(tiles)
            sim.load_pool(ranges, arrays)
            for i in range(n):
                row = sim.step(env[i], T[i], (18 + i) % 24, seeds[i])
                assert row.tobytes() == orc.step(env[i], T[i], (18 + i) % 24, seeds[i]).tobytes(), (tiles, i)
                if i in (2, n - 1):
                    ro, ao = orc.read_pool()
                    _same_pools(ro, sim.read_pool()[1], ao)
            assert sim.device_status() & 0xFF == 0
