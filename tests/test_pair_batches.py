"""Which batches run their FP64 passes as three paired launches (csrc/fdm.cuh: pair_batch_pays), on the CPU: the faster form
in batches that were measured both ways, and always three without an axis beyond 64 cells or with every member that long.
A small host program built with nvcc from the library's own header evaluates the rule."""
import os
import subprocess

import pytest

from les_impulse3d_64_b200 import _build

HARNESS = r'''
#include <cstdio>
#include <cstdlib>
#include "fdm.cuh"
using namespace cavity;
int main(int argc, char** argv) {
    std::vector<PairGrid> grids;
    for (int i = 1; i + 3 < argc; i += 4)
        for (int k = atoi(argv[i]); k > 0; k--) grids.push_back({atoi(argv[i + 1]), atoi(argv[i + 2]), atoi(argv[i + 3])});
    printf("%d\n", pair_batch_pays(grids));
    return 0;
}
'''


@pytest.fixture(scope='module')
def pays(tmp_path_factory):
    nvcc = _build.nvcc()
    if not os.path.exists(nvcc):
        pytest.skip('nvcc not found')
    d = tmp_path_factory.mktemp('pair_batches')
    (d / 'rule.cu').write_text(HARNESS)
    subprocess.run([nvcc, *_build.ARCH, '-std=c++17', f'-I{_build.ROOT / "include"}', f'-I{_build.CSRC}',
                    str(d / 'rule.cu'), '-o', str(d / 'rule')], check=True, capture_output=True)

    def run(*members):
        args = []
        for count, n in members:
            args += [count, *(n if isinstance(n, tuple) else (n, n, n))]
        return subprocess.run([str(d / 'rule'), *map(str, args)], check=True, capture_output=True,
                              text=True).stdout.strip() == '1'
    return run


@pytest.mark.parametrize('three', [
    [(4, 64), (1, 66)], [(8, 64), (1, 66)], [(32, 24), (1, 66)], [(96, 32), (1, 66)], [(128, 24), (1, 66)], [(16, 64), (4, 96)],
    [(24, 64), (8, 96)], [(24, 64), (1, (8, 8, 66))], [(7, 64), (1, (64, 64, 128))], [(16, 48), (2, 72)], [(8, 64), (1, 96)],
    [(6, 24), (6, 32), (6, 48), (6, 64), (1, 96)], [(4, 96), (4, 48)], [(48, 72), (1, 80)], [(200, 64)], [(300, 96)]])
def test_three_launches(pays, three):
    assert pays(*three)


@pytest.mark.parametrize('six', [
    [(12, 64), (1, 66)], [(24, 64), (1, 66)], [(48, 64), (1, 66)], [(24, 48), (1, 72)], [(48, 48), (1, 72)], [(24, 56), (1, 66)],
    [(24, 64), (2, 96)], [(24, 64), (4, 72)], [(48, 40), (1, 96)], [(24, 64), (1, (66, 66, 8))]])
def test_six_launches(pays, six):
    assert not pays(*six)
