"""The projection start with the residual of its guess in one launch against two launches (as tests/test_gpu_start.py), in
double: all fields of the FP64 form from checkpoints, with 4th- and 2nd-order edges.  Every value is formed by the same
expressions; the sums that the potential's mean comes from group their terms by other blocks, which is rounding: 1e-12 of a
field's largest value."""
import numpy as np
import pytest

from les_impulse3d_64_b200 import workloads
from les_impulse3d_64_b200.api import Batch, Cavity

pytestmark = pytest.mark.gpu


def double_fields(cav):
    """u, m, phi and the four potential increments of an FP64 cavity's checkpoint: parts of 256-byte multiples behind the
    header and the control block, before the statistics."""
    data = cav.checkpoint()
    nx, ny, nz = cav.nx, cav.ny, cav.nz
    faces = [(nx + 1) * ny * nz, nx * (ny + 1) * nz, nx * ny * (nz + 1)]
    sizes = faces + faces + [nx * ny * nz] * 5
    parts = [(8 * n + 255) // 256 * 256 for n in sizes + [6 * nx * ny]]
    at = len(data) - sum(parts)
    out = []
    for n, part in zip(sizes, parts):
        out.append(data[at:at + 8 * n].view(np.float64))
        at += part
    return out


@pytest.mark.parametrize('n, nz, options', [(16, 5, {}), (38, 8, dict(impulse_order=2)), (34, 33, dict(dt_lag=1)),
                                            (50, 9, dict(beta=1.4)), (58, 70, dict(phi_extrapolate=0)),
                                            (64, 64, dict(beta=1.5, impulse_order=2))])
def test_one_launch_equals_two_in_double(n, nz, options):
    s = workloads.settings(n, 500.0, nz=nz, cfl=0.5, **options)
    alone, member = Cavity(s), Cavity(s)
    batch = Batch([member], capacity=(1 << 18) // (n * n * nz) + 1)
    try:
        for cav in (alone, member):
            cav.initialize(*workloads.initial_noise(cav.shapes, 1e-2, 3))
        for _ in range(2):          # the second round starts from a full history
            alone.step_async(3)
            batch.step_async(3)
            assert alone.sync()['phi_passes'] == batch.sync()[0]['phi_passes']
        assert np.abs(double_fields(alone)[0] - alone.field('u').ravel()).max() < 1e-6
        for k, (x, y) in enumerate(zip(double_fields(alone), double_fields(member))):
            assert np.abs(x - y).max() <= 1e-12 * max(float(np.abs(y).max()), 1e-30), k
    finally:
        batch.close()
        alone.close()
        member.close()
