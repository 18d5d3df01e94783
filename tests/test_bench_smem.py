"""The delayed workloads' gathers are also rated against the shared memory that serves them."""
import bench


def test_shared_memory_roofline():
    r = bench.smem_roofline(1e12, 0.5)
    assert abs(r["achieved"] - 2000.0) < 1e-9 and abs(r["frac"] - r["achieved"] / r["peak"]) < 1e-12
    assert 3e4 < r["peak"] < 5e4   # 148 SMs x 128 B x 1.965 GHz = 37,228 GB/s


def test_delayed_workloads_report_it():
    groups = bench.c2_groups(15.0, sims_per_group=4)
    r = bench.batch_roofline(groups, 2.0)
    assert r["smem"]["achieved"] == r["achieved"] and r["smem"]["peak"] > r["peak"]
    c = bench.config_roofline(bench.c4_args(4, 4), 1000.0, True)
    assert c["smem"]["achieved"] == c["achieved"]
