"""The bench line's DRAM traffic per launch is the mean over the same launches
as its algorithmic bytes: full half-sweeps and a last one that gives labels."""


def test_mean_over_the_finest_levels_launches():
    import bench
    cfg = {"name": "hbp_1920x1080_L64_5lvl_x10_icm5"}
    one, two, ten = (bench.load_traffic(cfg, n) for n in (1, 2, 10))
    full = 2 * two - one
    assert abs(ten - (9 * full + one) / 10) <= 1e-9 * ten
    # Read and written: between what the messages kept in L2 leave and the algorithmic bytes.
    nodes = 1918 * 1078 // 2
    assert 0.85 < full / (nodes * 9 * 64 * 4) < 1.02
    assert 0.95 < one / (nodes * 5 * 64 * 4) < 1.05
    assert bench.load_traffic({"name": "another"}, 10) is None
