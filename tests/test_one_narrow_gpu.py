"""Calls around the sizes at which the narrow phase changes from one kernel to two:
the same edges give the same results in a call on either side of the limit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arms,g,rule", [(2, 5, 0), (2, 5, 1), (3, 33, 0), (3, 33, 2), (4, 32, 0), (4, 32, 3), (5, 64, 0),
                                         (5, 64, 2)])
def test_calls_around_the_one_kernel_limit(cuda, pkg, arms, g, rule):
    import numpy as np
    W = pkg.workloads
    rng = np.random.default_rng(100 * arms + g + rule)
    limit = 100000 // (arms * arms) * (2 if rule else 1)
    q0, q1 = W.random_edges(rng, limit + 1, arms, 4.0 if rule else 1.2)
    scene, robots = pkg.Scene(W.scene_config2(3)), pkg.RobotSet(arms, W.bases_facing_centre(arms, 0.71))
    a, b = cuda.from_numpy(q0).cuda(), cuda.from_numpy(q1).cuda()

    def run(s):
        return [t.cpu().numpy() for t in pkg.validate(scene, robots, a[s], b[s], g, rule=rule, range_=1.1)]

    two, one = run(slice(0, limit + 1)), run(slice(0, limit))
    prev = pkg.library().mrpop_set_fused_edges(1 << 30)
    try:
        fused = run(slice(0, limit + 1))
    finally:
        pkg.library().mrpop_set_fused_edges(prev)
    for x, y, z in zip(two, one, fused):
        assert np.array_equal(x[:limit], y) and np.array_equal(x, z)
    assert 0 < two[0].sum() < limit
    assert scene.status() == 0
