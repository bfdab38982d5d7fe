"""Pools that come from outside hold what no step leaves behind: state bytes
that do not match the ranges, larvae in their first day. Every route of a
step gives the same records for them, the oracle's."""
import ctypes as C

import numpy as np
import pytest

from tests.test_step_paths import _same_pools, _workload

pytestmark = pytest.mark.gpu


def _run_and_compare(ranges, arrays, T, env, seeds, cc, calls, tiles):
    """`calls` runs of so many hours each, against the oracle's rows and final pool."""
    from oracle import OracleSim
    from sampo_gb300.sim import Simulation
    cap, n = 1 << 20, sum(calls)
    orc = OracleSim(cap)
    orc.load_pool(ranges, arrays)
    with Simulation(capacity=cap, carrying_capacity=cc, max_steps=n + 1) as sim:
        sim.set_inputs(T[:n], env[:n])
        sim.set_seeds(0, seeds[:n])
        sim.set_small_step(tiles)
        sim.load_pool(ranges, arrays)
        rows = np.concatenate([sim.run(c) for c in calls])
        assert sim.device_status() & 0xFF == 0
        pop, pool = sim.read_pool()
    for i in range(n):
        assert rows[i].tobytes() == orc.step(env[i], T[i], i % 24, seeds[i]).tobytes(), f"step {i}"
    ro, ao = orc.read_pool()
    assert np.array_equal(np.asarray(pop["ranges"], np.int64), np.asarray(ro, np.int64))
    _same_pools(ro, pool, ao)
    return ro, pool


@pytest.mark.parametrize("tiles", [0, None])
@pytest.mark.parametrize("free", [False, True])
@pytest.mark.parametrize("calls", [(1,), (5,), (24, 2)])
def test_state_bytes_follow_the_ranges(gpu_ready, oracle_mod, tiles, free, calls):
    """State bytes of other states: a step writes the state of the range an
    agent is in, for those that stay as for those that move on."""
    ranges, arrays, T, env, seeds = _workload((1300, 900, 300, 700), 30, 30000.0, seed=4)
    arrays["state"][:] = (arrays["state"] * 3 + 5) % 8
    if free:  # records that are moved whole
        s, e = int(ranges[0][0]), int(ranges[0][1])
        arrays["numEggBatches"][s:e:3] = 5
    ro, pool = _run_and_compare(ranges, arrays, T, env, seeds, 30000.0, calls, tiles)
    for k in range(8):
        assert np.all(pool["state"][int(ro[k][0]):int(ro[k][1])] == k), k


@pytest.mark.parametrize("eggs", [2000, 420000])
def test_state_bytes_of_caller_owned_pools(gpu_ready, eggs):
    """The same through sampo_step_noalloc, one launch and three."""
    torch = pytest.importorskip("torch")
    from sampo_gb300 import _lib, inputs
    from sampo_gb300.population import make_pool
    from sampo_gb300.sim import pop_from_ranges, seed_stream
    from tests.test_zz_no_alloc import _device_pool, _download, _upload
    cc, T, cap = 4000.0, np.array([29.0], np.float32), 1 << 20
    env = np.zeros(1, dtype=inputs.ENV_DTYPE)
    env["bloodmealSuccess"] = 0.5
    env["carryingCapacity"] = cc
    ranges, arrays = make_pool((eggs, 90000, 20000, 50000), T[0], seed=7)
    arrays["state"][:] = (arrays["state"] + 1) % 8
    tin, din = _device_pool(torch, cap)
    tout, dout = _device_pool(torch, cap)
    _upload(torch, tin, ranges, arrays)
    torch.cuda.synchronize()
    p, e = pop_from_ranges(ranges), _lib.Environment(*[float(env[0][k]) for k in inputs.ENV_DTYPE.names])
    s = np.ascontiguousarray(seed_stream(3, 1)[1][0], dtype=np.uint32)
    row, out, bnc = _lib.StatsRow(), _lib.Population(), _lib.BitesCycles()
    assert _lib.load().sampo_step_noalloc(C.byref(din), cap, C.byref(dout), cap, C.byref(p), C.byref(e), float(T[0]), 19,
                                          s.ctypes.data, cc, C.byref(row), C.byref(out), C.byref(bnc), 0, None) == 0
    got = _download(tout, int(out.r[7].end))
    for k in range(8):
        assert np.all(got["state"][out.r[k].start:out.r[k].end] == k), k


@pytest.mark.parametrize("tiles", [0, None])
@pytest.mark.parametrize("ages", [(0,), (0, 700), (21,), (5, 30)])
def test_larvae_younger_than_a_day(gpu_ready, oracle_mod, tiles, ages):
    """A larva hatches at 24 hours, but a pool may bring younger ones: with
    hoursInState = age - 24 their records follow from their state, and their
    day, the 0th, has its mortality like the others."""
    ranges, arrays, T, env, seeds = _workload((700, 2100, 300, 700), 30, 30000.0, seed=6)
    s, e = int(ranges[1][0]), int(ranges[1][1])
    arrays["ageInHours"][s:e] = np.resize(np.array(ages, np.float32), e - s)
    arrays["hoursInState"][s:e] = arrays["ageInHours"][s:e] - np.float32(24.0)
    _run_and_compare(ranges, arrays, T, env, seeds, 30000.0, (26, 4), tiles)


def test_batch_with_a_pool_of_whole_records(gpu_ready, tmp_path):
    """A slot resumed from a pool with free records makes its batch move whole
    records (three kernels an hour) until it is removed; the replicates beside
    it, which decide ahead before and after (one count pass a day), and the
    slot itself equal their plain runs."""
    import dataclasses
    from sampo_gb300.batch import Batch, admit
    from sampo_gb300.sim import Simulation
    from tests.test_batch import SPECS, compare
    n, cc, cap = 30, 30000.0, 1 << 18
    ranges, arrays, T, env, seeds = _workload((9000, 7000, 2000, 5000), n, cc, seed=8)
    s, e = int(ranges[1][0]), int(ranges[1][1])
    arrays["hoursInState"][s:e:2] += np.float32(0.25)
    ck = str(tmp_path / "whole.ck")
    with Simulation(capacity=cap, carrying_capacity=cc, max_steps=n + 1) as sim:
        sim.set_inputs(T, env)
        sim.set_seeds(0, seeds)
        sim.load_pool(ranges, arrays)
        sim.checkpoint(ck)
        sim.run(n)
        want, (pop, pool) = sim.current_row(), sim.read_pool()
    big = dataclasses.replace(SPECS[4], initial=90000, days=6, capacity=1800000)
    small = dataclasses.replace(SPECS[1], days=6)
    with Batch(max_replicates=4, ring_steps=150) as b:
        slots = [admit(b, x, 144) for x in (big, small)]

        def kernels(hours):
            before = b.launches()
            b.run(hours)
            return b.launches() - before

        assert kernels(24) == 1 + 50          # count, publish, 24 x (scatter, publish)
        w = b.add(cap, cc, stop_step=n)
        b.set_inputs(w, T, env)
        b.set_seeds(w, 0, seeds)
        b.resume(w, ck)
        assert kernels(24) == 1 + 72
        late = admit(b, small, 72)            # admitted into whole records
        assert kernels(24) == 1 + 72
        assert b.rows(w, n, 1)[0].tobytes() == want.tobytes()
        bpop, bpool = b.read_pool(w)
        assert np.array_equal(bpop["ranges"], pop["ranges"])
        _same_pools(pop["ranges"], bpool, pool)
        b.remove(w)
        assert kernels(72) == 1 + 150
        compare(b, slots[0], big, 144, "large replicate")
        compare(b, slots[1], small, 144, "small replicate")
        compare(b, late, small, 72, "late replicate")
