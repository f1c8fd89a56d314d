"""The projection start and the residual of its guess as one launch (fused_start_kernel, at most 2^18 cells in all)
against two launches: a cavity alone, and the same cavity in a batch whose slots hold more cells than that."""
import numpy as np
import pytest

from les_impulse3d_64_b200 import workloads
from les_impulse3d_64_b200.api import Batch, Cavity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
@pytest.mark.parametrize('n, nz, options', [(16, 5, {}), (32, 8, {}), (34, 33, dict(dt_lag=1)), (50, 9, dict(beta=1.4)),
                                            (58, 70, dict(phi_extrapolate=0)), (64, 64, dict(beta=1.5))])
def test_one_launch_equals_two(n, nz, options, precision):
    """Every value is formed by the same expressions; the sums group their terms by other blocks, and through the
    potential's mean that is rounding: 1e-12 in FP64, 1e-6 in the FP32 fields of the mixed form."""
    s = workloads.settings(n, 500.0, nz=nz, cfl=0.5, **options)
    alone, member = Cavity(s, precision=precision), Cavity(s, precision=precision)
    batch = Batch([member], capacity=(1 << 18) // (n * n * nz) + 1)
    try:
        for cav in (alone, member):
            cav.initialize(*workloads.initial_noise(cav.shapes, 1e-2, 3))
        for _ in range(2):          # the second round starts from a full history
            alone.step_async(3)
            batch.step_async(3)
            a, b = alone.sync(), batch.sync()[0]
            assert a['steps'] == b['steps'] and a['phi_passes'] == b['phi_passes']
        for k in ('u', 'v', 'w', 'mx', 'my', 'mz', 'phi'):
            x, y = alone.field(k), member.field(k)
            tol = 1e-12 if precision == 'fp64' and k == 'phi' else 1e-6
            assert np.abs(x - y).max() <= tol * max(float(np.abs(y).max()), 1e-30), k
    finally:
        batch.close()
        alone.close()
        member.close()
