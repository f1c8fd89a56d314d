"""cavity_sweep_kernel names the sweep kernel that the library's own rules chose; the bench line's roofline shows it."""
import pytest

import bench
from les_impulse3d_64_b200 import workloads
from les_impulse3d_64_b200.api import Cavity

pytestmark = pytest.mark.gpu


def test_the_name_of_the_running_sweep(monkeypatch):
    for key in ('CAVITY_SWEEP', 'CAVITY_COLUMN', 'CAVITY_TUNE_FILE'):
        monkeypatch.delenv(key, raising=False)

    def name(precision, n, **env):
        for key, value in env.items():
            monkeypatch.setenv(key, value)
        cav = Cavity(workloads.settings(n, 500.0, nz=16), precision=precision)
        for key in env:
            monkeypatch.delenv(key)
        try:
            return bench.sweep_kernel_name(precision, cav)
        finally:
            cav.close()

    assert name('fp64', 24) == 'sweep_tile_kernel'
    assert name('mixed', 24) == 'sweep_pair_kernel'
    assert name('mixed', 24, CAVITY_COLUMN='2') == 'sweep_column_kernel'
    assert name('mixed', 256) == 'sweep_column_kernel'
    assert name('mixed', 256, CAVITY_COLUMN='0') == 'sweep_pair_kernel'
    for kind, kernel in (('tile', 'sweep_tile_kernel'), ('march', 'sweep_march_kernel'), ('face', 'momentum_kernel')):
        assert name('mixed', 24, CAVITY_SWEEP=kind) == kernel
