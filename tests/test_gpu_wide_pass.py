"""The paired FP64 pass on axes of 65 to 128 cells (pair_wide_kernel, csrc/fdm.cuh): bit for bit the six-launch pass at the
edges of its tiles and panels, alone and in a batch with smaller members."""
import os

import numpy as np
import pytest

from les_impulse3d_64_b200 import workloads
from les_impulse3d_64_b200.api import load_library
from les_impulse3d_64_b200.ensemble import Ensemble
from test_gpu_fdm import call_fdm, fdm_reference, random_operands

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dims', [(65, 64, 5), (64, 65, 7), (6, 7, 65), (66, 33, 128), (96, 96, 96), (100, 100, 75),
                                  (127, 128, 9), (128, 127, 66), (8, 128, 17), (128, 9, 64)])
def test_wide_pass_equals_six_launches(dims, monkeypatch):
    lib = load_library()
    S, il, r, phi = random_operands(*dims, seed=sum(dims) + 41)
    monkeypatch.setenv('CAVITY_FDM_FUSED', '2')
    out = call_fdm(lib, 'cavity_fdm_pass', S, il, r, phi)
    monkeypatch.setenv('CAVITY_FDM_FUSED', '0')
    assert np.array_equal(call_fdm(lib, 'cavity_fdm_pass', S, il, r, phi), out)
    ref = fdm_reference(S, r, il, phi)
    assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_wide_batch_equals_six_launches(precision):
    """Members of 24, 66 and 64 x 64 x 100 cells: every phase by the streamed kernel, against six launches."""
    cases = workloads.ensemble_cases(count=3, seed=31, sizes=(24, 66), re_range=(100.0, 2000.0))
    cases[0]['settings'] = workloads.settings(66, 900.0, nz=18, beta=1.4, cfl=0.5)
    cases[1]['settings'] = workloads.settings(64, 700.0, nz=100, cfl=0.5)
    for c in cases:
        c['precision'] = precision

    def run(form):
        old = os.environ.pop('CAVITY_FDM_FUSED', None)
        if form is not None:
            os.environ['CAVITY_FDM_FUSED'] = form
        try:
            ens = Ensemble(cases, group='precision')
        finally:
            os.environ.pop('CAVITY_FDM_FUSED', None)
            if old is not None:
                os.environ['CAVITY_FDM_FUSED'] = old
        try:
            assert len(ens.batches) == 1
            ens.advance(3, chunk=3)
            return [ens.fields(i) for i in range(len(cases))]
        finally:
            ens.close()

    wide, six = run(None), run('0')
    for i in range(len(cases)):
        for k in wide[i]:
            assert np.array_equal(wide[i][k], six[i][k]), (i, k)
