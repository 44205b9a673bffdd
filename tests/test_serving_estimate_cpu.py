"""The serving loop's memory estimate is an upper one: against the bytes engines were seen to hold
(fcw_info.device_bytes on folded icospheres, cap fraction 0.1), plus the sources and records of a job
that runs every vertex, and not so far above them that jobs wait for memory that is there."""
import pytest

from fastcorticalwiring_b200 import serving as S

# vertices, faces, block_k, depth, options, engine bytes
HELD = [
    (2306, 4551, 64, 1, {}, 28_809_863),
    (9218, 18322, 64, 1, {}, 120_410_097),
    (36866, 73491, 64, 1, {}, 505_801_794),
    (147458, 294471, 64, 1, {}, 2_094_541_301),
    (147458, 294471, 64, 1, dict(tc_sweeps=1, refine=2), 2_499_060_225),
    (589826, 1178700, 64, 1, {}, 8_673_428_299),
    (589826, 1178700, 64, 1, dict(tc_sweeps=1, refine=2), 10_423_707_663),
    (9218, 18322, 1024, 4, {}, 3_284_161_062),
    (147458, 294471, 1024, 4, {}, 53_610_751_190),
    (589826, 1178700, 1024, 3, {}, 163_289_929_430),
]


@pytest.mark.parametrize("n,nf,k,depth,opts,held", HELD)
def test_estimate_covers_what_engines_hold(n, nf, k, depth, opts, held):
    stride = S._stride(12, 3)
    need = held + n * (4 + 8 * stride)
    est = S.estimate_device_bytes(n, 2 * n, k, depth, n, stride, **opts)
    assert need <= est <= 1.3 * need + (64 << 20)


def test_server_passes_its_engine_options():
    srv = object.__new__(S.Server)
    job = S.Job("a", None, None, [True] * 100_000, scales=(0.01, 0.02), sources=[1, 2, 3])
    est = []
    for extra in ({}, dict(tc_sweeps=1), dict(refine=1), dict(leaf_size=256)):
        srv.params = dict(block_k=64, pipeline_depth=1, **extra)
        est.append(srv._estimate(S._Pending(job, 0.0)))
    assert min(est[1:]) > est[0]
