"""The packed sweep's walk up columns (sweep_column.cuh) gives the packed tile sweep's step bit for bit: grids that cut its
16 x 16 columns, chunks of every kind (one layer pair, an upper half outside the box, the longest), 2nd-order stencils,
walls inside a chunk, and a batch of several sizes."""
import os

import numpy as np
import pytest

from cases import base_settings
from les_impulse3d_64_b200 import workloads
from les_impulse3d_64_b200.ensemble import Ensemble
from test_gpu_sweep import FIELDS, GRIDS, run

pytestmark = pytest.mark.gpu

MORE = [
    dict(nx=18, ny=18, nz=6),                                        # columns of two cells
    dict(nx=50, ny=50, nz=37, grid_stretch=1, grid_dx_wall=0.008),
    dict(nx=34, ny=34, nz=150, impulse_order4_ramp=2.0),             # beyond one chunk of the longest
    dict(nx=96, ny=96, nz=33),                                       # tiles without walls
]


@pytest.mark.parametrize('chunks', ['1', '3', '200'])
@pytest.mark.parametrize('grid', range(len(GRIDS) + len(MORE)))
def test_column_equals_tile(grid, chunks):
    s = base_settings(adaptive_dt=1, dt_max=0.01, nu=0.002, lid_ramp_t=0.5, **(GRIDS + MORE)[grid])
    rc, fc = run(s, 'mixed', {'CAVITY_COLUMN': chunks})
    rt, ft = run(s, 'mixed', {'CAVITY_COLUMN': '0'})
    assert rc == rt
    for k in FIELDS:
        assert np.array_equal(fc[k], ft[k]), k


def test_column_batch_equals_tile():
    cases = workloads.ensemble_cases(count=3, seed=37, sizes=(24, 40), re_range=(100.0, 2000.0))
    cases[0]['settings'] = workloads.settings(50, 900.0, nz=18, beta=1.4, cfl=0.5)
    for c in cases:
        c['precision'] = 'mixed'

    def fields(column):
        old = os.environ.pop('CAVITY_COLUMN', None)
        os.environ['CAVITY_COLUMN'] = column
        try:
            ens = Ensemble(cases, group='precision')
        finally:
            os.environ.pop('CAVITY_COLUMN', None)
            if old is not None:
                os.environ['CAVITY_COLUMN'] = old
        try:
            assert len(ens.batches) == 1
            ens.advance(3, chunk=3)
            return [ens.fields(i) for i in range(len(cases))]
        finally:
            ens.close()

    tile = fields('0')
    for column in ('1', '4'):
        for a, b in zip(fields(column), tile):
            for k in b:
                assert np.array_equal(a[k], b[k]), (column, k)
