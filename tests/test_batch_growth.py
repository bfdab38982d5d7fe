"""Replicates that are moved into other buffers (sampo_batch_grow) while their
batch decides hours ahead go on exactly as the plain run with room to spare."""
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
