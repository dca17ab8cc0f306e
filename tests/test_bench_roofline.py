"""The DRAM bytes beside a roofline are averaged the way its algorithmic bytes and durations are."""
from __future__ import annotations


def test_average_traffic_of_alternating_launches():
    import bench
    full, _ = bench.profile_traffic('cocg_stencil_c128', 'aniso_blocks')
    mean, source = bench.profile_traffic('cocg_stencil_c128', 'aniso_blocks', average=True)
    from meanas_b200 import workloads
    p = workloads.BY_NAME['aniso_blocks']()
    alg = bench.kernel_bytes(0, p) * p.n_cells
    # 288 B per cell on average, 360 with the x updates; traffic is within 10 % of either
    assert abs(mean / alg - 1) < 0.1 and abs(full / (alg * 360 / 288) - 1) < 0.1
    assert source.startswith('profiles/cocg_stencil_c128_aniso160.md')
    # a file with one kind of launch has one figure
    assert bench.profile_traffic('bicgstab_P_c64', 'aniso_blocks', average=True) == \
        bench.profile_traffic('bicgstab_P_c64', 'aniso_blocks')
