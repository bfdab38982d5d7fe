"""Replicates that are moved into other buffers (sampo_batch_grow) while their
batch decides hours ahead go on exactly as the plain run with room to spare:
whichever hour of a run a pause falls on, in their slots or through a
checkpoint in another batch."""
import ctypes as C
import dataclasses
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _specs(scale, capacity):
    """A replicate that outgrows `capacity` and, to have the batch decide ahead, a large one beside it."""
    from sampo_gb300.batch import ReplicateSpec
    tight = ReplicateSpec(initial=2000 * scale, seed=21, mean_t=29.0, amplitude=2.0, rain_mean=3.0, days=16, capacity=capacity)
    beside = ReplicateSpec(initial=120000, seed=15, mean_t=28.0, amplitude=4.0, rain_mean=3.0, days=16, capacity=2400000)
    return tight, beside


@pytest.mark.parametrize("hours", [49, 50, 51])
def test_shrunk_pools_move_into_smaller_buffers(gpu_ready, hours):
    """A pool that has shrunk, moved into buffers of its size after runs that
    decided ahead (with the span counts in each of their three sets): the
    batch goes on deciding ahead and the inputs that lie behind the span
    arrays stay what they were."""
    from sampo_gb300.batch import Batch, ReplicateSpec, admit
    from tests.test_batch import plain_run
    spec = ReplicateSpec(initial=300000, seed=31, mean_t=17.0, amplitude=1.0, rain_mean=4.0, days=8, capacity=3000000, age_days_max=-1)
    _, beside = _specs(1, 4096)
    n = spec.steps
    want = plain_run(spec, n)[0]
    with Batch(max_replicates=2, ring_steps=n + 1) as b:
        s, t = admit(b, spec, n), admit(b, beside, n)
        b.run(hours)
        end = int(b.states()[s]["end"])
        assert end < 260000  # (a tenth of the eggs dies a day: about 243,000)
        b.grow(s, end)
        for _ in range(4 * n):
            st = b.states()[s]
            if int(st["step"]) == n:
                break
            if not st["active"]:
                assert st["status"] == 1, st
                b.grow(s, max(int(st["end"]), int(st["capacity"]) + 1024))
            b.run(min(24, n - int(st["step"])))
        assert b.rows(s, 0, n + 1).tobytes() == want.tobytes()
        m = int(b.states()[t]["step"])
        assert b.rows(t, 0, m + 1).tobytes() == plain_run(beside, m)[0].tobytes()


def _pause_step(rows, capacity):
    """The first step whose next layout passes `capacity` (rows of the run with room to spare)."""
    return int(np.argmax(rows["ranges"][:, 7, 1] > capacity)) - 1


@pytest.mark.parametrize("scale,capacity", [(1, 4096), (20, 90000)])
@pytest.mark.parametrize("where", ["first hour", "within", "last hour", "single hour"])
def test_checkpoint_after_a_pause(gpu_ready, tmp_path, scale, capacity, where):
    """A paused replicate's device seed stream is as it was: the checkpoint
    taken after sampo_batch_grow holds every seed the coming steps need."""
    from sampo_gb300._lib import Population, SampoError
    from sampo_gb300.batch import Batch, admit
    from tests.test_batch import plain_run
    tight, beside = _specs(scale, capacity)
    n = tight.steps
    want = plain_run(dataclasses.replace(tight, capacity=400000 * scale), n)[0]
    p = _pause_step(want, capacity)
    assert 24 < p < n - 24
    ck = str(tmp_path / "slot.ck")
    with Batch(max_replicates=2, ring_steps=n + 1) as b:
        s = admit(b, tight, n, device_seeds=True)
        if scale > 1:
            admit(b, beside, n, device_seeds=True)
        before, hours = {"first hour": (p, 24), "within": (p - 9, 24), "last hour": (p - 23, 24), "single hour": (p, 1)}[where]
        b.run(before)
        b.run(hours)
        step, active, bits = b.state(s)
        assert (step, active, bits) == (p, False, 1)
        assert b.seed_state(s)[1] == p + 1
        b.grow(s, 400000 * scale)
        b.checkpoint(s, ck)
        b.run(n - p)
        assert b.rows(s, 0, n + 1).tobytes() == want.tobytes(), "in its slot"
    raw = bytearray(open(ck, "rb").read())
    # the first step whose seeds the file's stream has not drawn
    at = len(b"SAMPOCK1") + 12 + C.sizeof(Population) + 16 + 8 + C.sizeof(Population)
    assert struct.unpack_from("<I", raw, at)[0] == p + 1
    struct.pack_into("<I", raw, at, p + 2)
    open(ck + ".bad", "wb").write(bytes(raw))
    T, env = tight.inputs()
    with Batch(max_replicates=1, ring_steps=n + 1) as b:
        s = b.add(400000 * scale, tight.cc, stop_step=n)
        b.set_inputs(s, T[:n], env[:n])
        with pytest.raises(SampoError):  # a file without the seeds of step p
            b.resume(s, ck + ".bad")
        b.resume(s, ck)
        b.run(n - p)
        assert b.rows(s, p, n + 1 - p).tobytes() == want[p:].tobytes(), "from its checkpoint"
