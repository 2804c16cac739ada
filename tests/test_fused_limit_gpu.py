"""The largest calls that run as one fused launch: a limit set by
mrpop_set_fused_edges holds for calls of every rule, the default one lets
segmented calls be larger.  The launch form shows in the kernel times (a split
call launches broad kernels)."""
import pytest

pytestmark = pytest.mark.gpu


def _is_fused(cuda, pkg, arms, n, rule, g=4):
    import numpy as np
    W = pkg.workloads
    bases = W.bases_facing_centre(arms, 0.71)
    q0, q1 = W.random_edges(np.random.default_rng(n), n, arms, 2.0)
    scene, robots = pkg.Scene(W.scene_config2(3)), pkg.RobotSet(arms, bases)
    a, b = cuda.from_numpy(q0).cuda(), cuda.from_numpy(q1).cuda()
    cuda.cuda.synchronize()
    pkg.kernel_timing(True)
    try:
        pkg.kernel_times()
        pkg.validate(scene, robots, a, b, g, rule=rule, range_=1.0 if rule else 0.0)
        cuda.cuda.synchronize()
        t = pkg.kernel_times()
    finally:
        pkg.kernel_timing(False)
    assert t["broad"][0] or t["fused"][0]
    return t["broad"][0] == 0


@pytest.mark.parametrize("rule", [0, 1, 2, 3])
@pytest.mark.parametrize("limit", [1, 700, 2049])
def test_a_limit_set_holds_for_every_rule(cuda, pkg, limit, rule):
    lib = pkg.library()
    prev = lib.mrpop_set_fused_edges(limit)
    try:
        assert _is_fused(cuda, pkg, 2, limit, rule)
        assert not _is_fused(cuda, pkg, 2, limit + 1, rule)
        assert not _is_fused(cuda, pkg, 2, 2 * limit, rule)
    finally:
        assert lib.mrpop_set_fused_edges(prev) == limit


@pytest.mark.parametrize("setting", [0, 2048])
def test_default_limits(cuda, pkg, setting):
    lib = pkg.library()
    prev = lib.mrpop_set_fused_edges(setting)
    try:
        for rule, limit in ((0, 2048), (1, 5120), (2, 5120), (3, 5120)):
            assert _is_fused(cuda, pkg, 2, limit, rule)
            assert not _is_fused(cuda, pkg, 2, limit + 1, rule)
    finally:
        assert lib.mrpop_set_fused_edges(prev) == 2048


@pytest.mark.parametrize("arms,limit", [(1, 5120), (3, 5120), (4, 5120), (5, 4096)])
def test_default_limit_of_segmented_calls_by_arms(cuda, pkg, arms, limit):
    lib = pkg.library()
    prev = lib.mrpop_set_fused_edges(0)
    try:
        for rule in (1, 2, 3):
            assert _is_fused(cuda, pkg, arms, limit, rule)
            assert not _is_fused(cuda, pkg, arms, limit + 1, rule)
    finally:
        lib.mrpop_set_fused_edges(prev)


@pytest.mark.parametrize("arms,g,limit", [(1, 32, 2048), (3, 32, 2048), (4, 32, 1280), (4, 33, 2048), (5, 1, 512),
                                          (5, 32, 512), (5, 33, 2048)])
def test_default_limit_of_single_segment_calls_by_arms(cuda, pkg, arms, g, limit):
    lib = pkg.library()
    prev = lib.mrpop_set_fused_edges(0)
    try:
        assert _is_fused(cuda, pkg, arms, limit, 0, g)
        assert not _is_fused(cuda, pkg, arms, limit + 1, 0, g)
    finally:
        lib.mrpop_set_fused_edges(prev)


@pytest.mark.parametrize("arms,n,shelf", [(4, 1281, False), (5, 513, False), (5, 2048, False), (5, 1025, True)])
def test_calls_above_the_lower_limits_equal_fused_ones(cuda, pkg, arms, n, shelf):
    import numpy as np
    W = pkg.workloads
    bases = W.bases_config2() if arms == 4 else W.bases_config3()
    q0, q1 = W.random_edges(np.random.default_rng(n), n, arms, 1.5)
    # (with 5 arms the bin table is in every edge's way: all of them collide)
    scene = pkg.Scene(W.scene_config3(3) if shelf else W.scene_config2(3))
    robots = pkg.RobotSet(arms, bases)
    a, b = cuda.from_numpy(q0).cuda(), cuda.from_numpy(q1).cuda()
    lib, out = pkg.library(), []
    for limit in (0, 1 << 30):
        prev = lib.mrpop_set_fused_edges(limit)
        try:
            out.append([t.cpu().numpy() for t in pkg.validate(scene, robots, a, b, 31)])
        finally:
            lib.mrpop_set_fused_edges(prev)
    if arms == 4 or shelf:
        assert 0 < int(out[0][0].sum()) < n
    assert all(np.array_equal(x, y) for x, y in zip(*out))
