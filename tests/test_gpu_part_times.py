"""cavity_batch_part_times on a batch with empty slots: the instrumented graphs record a member in their place, as the plain
ones do, and the steps are ordinary ones; a batch of empty slots alone is refused."""
import numpy as np
import pytest

from les_impulse3d_64_b200 import workloads
from les_impulse3d_64_b200.api import Batch, Cavity

pytestmark = pytest.mark.gpu


def make(seed):
    cav = Cavity(workloads.settings(24, 400.0, nz=13, beta=1.3, cfl=0.5), precision='mixed')
    cav.initialize(*workloads.initial_noise(cav.shapes, 1e-2, seed))
    return cav


def test_part_times_with_empty_slots():
    a, b = [make(1), make(2)], [make(1), make(2)]
    timed, plain = Batch(a, capacity=4), Batch(b, capacity=4)
    try:
        for batch in (timed, plain):               # slot 0 empty too
            batch.set_member(0, None)
        times = timed.part_times(2)
        assert all(t > 0 for t in times.values())
        plain.step_async(2)
        plain.sync()
        for batch, c in ((timed, a), (plain, b)):
            batch.set_member(0, c[0])
            batch.step_async(2)
            batch.sync()
        for x, y in zip(a, b):
            assert x.report() == y.report()
            for k in ('u', 'v', 'w', 'mx', 'my', 'mz', 'phi'):
                assert np.array_equal(x.field(k), y.field(k)), k
        for slot in range(2):
            timed.set_member(slot, None)
        with pytest.raises(RuntimeError, match='every slot is empty'):
            timed.part_times(1)
    finally:
        timed.close()
        plain.close()
        for cav in a + b:
            cav.close()
