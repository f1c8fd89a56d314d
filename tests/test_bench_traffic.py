"""The bench line's DRAM traffic is that of the sweep kernel it names: of the profile whose title holds the kernel, none
where no profile of the workload does."""
import bench


def test_traffic_belongs_to_the_kernel(tmp_path, monkeypatch):
    folder = tmp_path / 'profiles'
    folder.mkdir()
    (folder / 'momentum_sweep_w.md').write_text('# sweep_tile_kernel<float>, W\n\ntraffic_bytes_per_launch: 80\n')
    (folder / 'momentum_sweep_column_w.md').write_text('# sweep_column_kernel<16, 16>, W\ntraffic_bytes_per_launch: 75\n')
    (folder / 'momentum_sweep_pair_w.md').write_text('# sweep_pair_kernel<8> against sweep_tile_kernel<float>, W\n')
    monkeypatch.setattr(bench, 'ROOT', tmp_path)
    assert bench.profile_traffic('w', 'sweep_tile_kernel') == 80
    assert bench.profile_traffic('w', 'sweep_column_kernel') == 75
    assert bench.profile_traffic('w', 'sweep_pair_kernel') is None
    assert bench.profile_traffic('v', 'sweep_tile_kernel') is None


def test_committed_profiles():
    for workload, kernel in (('c2_64cube_re1000', 'sweep_tile_kernel'), ('c3_128cube_re3200', 'sweep_column_kernel')):
        assert bench.profile_traffic(workload, kernel) > 1e6
