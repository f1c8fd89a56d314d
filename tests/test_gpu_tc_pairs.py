"""The mixed form's pressure pass as three launches of two chained tcgen05 transforms (csrc/tc_pair.cuh, the default
where no axis exceeds 256 cells): against the FP64 transforms at the edges of its tiles, panels and rings, and in a
batch of several sizes against the members alone."""
import ctypes as ct

import numpy as np
import pytest

from les_impulse3d_64_b200 import workloads
from les_impulse3d_64_b200.api import load_library
from les_impulse3d_64_b200.ensemble import Ensemble
from test_gpu_fdm import call_fdm, fdm_reference, random_operands

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dims', [(4, 4, 1), (8, 6, 32), (32, 32, 33), (100, 100, 75), (128, 128, 128), (128, 129, 16),
                                  (132, 132, 31), (160, 96, 65), (192, 193, 20), (256, 256, 9), (16, 256, 24),
                                  (8, 8, 256)])
def test_pass_matches_numpy(dims):
    """Tolerance: a product accumulates 3 K / 8 partial sums in FP32, each rounded towards zero (2^-23), and a pass has
    six products: 6 * 3 K / 8 * 2^-23 of the update's largest entry bounds what the roundings can add up to."""
    lib = load_library()
    lib.cavity_last_error.restype = ct.c_char_p
    S, il, r, phi = random_operands(*dims, seed=sum(dims) + 23)
    out = call_fdm(lib, 'cavity_fdm_pass_tf32', S, il, r, phi)
    upd = fdm_reference(S, r, il, np.zeros_like(phi))
    k = max(32, *dims)
    assert np.abs(out - phi - upd).max() <= 6 * (3 * k / 8) * 2.0 ** -23 * np.abs(upd).max()


def test_batch_of_several_sizes_matches_alone(monkeypatch):
    """Members of several sizes share one variant of the kernels: each ends equal to itself alone to rounding (1e-6 in
    the FP32 fields; the column kernels' reductions group their sums differently in a batch)."""
    monkeypatch.setenv('CAVITY_FDM', 'tc')
    cases = workloads.ensemble_cases(count=4, seed=29, sizes=(16, 40), re_range=(100.0, 2000.0))
    cases[0]['settings'] = workloads.settings(132, 800.0, nz=9, cfl=0.5)
    ens = Ensemble(cases, group='precision')
    try:
        assert len(ens.batches) == 1
        ens.advance(3, chunk=3)
        together = [ens.fields(i) for i in range(len(cases))]
    finally:
        ens.close()
    for i in range(len(cases)):
        alone = Ensemble([cases[i]], batched=False)
        try:
            alone.advance(3, chunk=1)
            f = alone.fields(0)
        finally:
            alone.close()
        for k in f:
            err = float(np.abs(f[k] - together[i][k]).max() / max(np.abs(f[k]).max(), 1e-30))
            assert err <= 1e-6, (i, k, err)
