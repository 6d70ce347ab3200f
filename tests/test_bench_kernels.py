"""bench.py names the kernel that the tuner chose for the ladder, and gives the
committed capture's traffic for that kernel alone."""
import bench


def launch(**kw):
    return dict(dict(bn=192, sps=2, pairs=3, M=51360, N=528, K=51360), **kw)


def test_ladder_kernel_and_traffic_follow_the_tuner():
    assert bench.tc_kernel(launch()) == "gemm_tc_kernel<192, 0, 2>"
    assert bench.tc_kernel(launch(bn=256, sps=1)) == "gemm_tc_kernel<256, 0, 1>"
    assert bench.tc_kernel(launch(bn=256)) == "gemm_pair_kernel<2>"
    assert bench.tc_kernel(launch(bn=256, pairs=6)) == "gemm_pair_kernel<3>"
    traffic, source = bench.ladder_traffic(launch())
    assert traffic == bench.ncu_traffic() and traffic > 0 and "not measured in this run" in source
    for other in (launch(bn=256), launch(bn=256, sps=1), launch(M=1275, N=18145)):
        traffic, source = bench.ladder_traffic(other)
        assert traffic is None and source.startswith("not measured")
