"""Segmented calls around the sizes at which they change from one fused launch to
segment rounds of the split kernels: the same edges give the same results on
both sides, and alone in either form."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rule", [1, 2, 3])
@pytest.mark.parametrize("n", [2048, 2049, 5120, 5121])
def test_segmented_calls_around_the_fused_limit(cuda, pkg, rule, n):
    import numpy as np
    W = pkg.workloads
    rng = np.random.default_rng(n + rule)
    bases = W.bases_facing_centre(2, 0.71)
    q0, q1 = W.random_edges(rng, n, 2, 4.0)
    scene, robots = pkg.Scene(W.scene_config2(3)), pkg.RobotSet(2, bases)
    a, b = cuda.from_numpy(q0).cuda(), cuda.from_numpy(q1).cuda()
    lib = pkg.library()
    out = []
    for limit in (0, -1, 1 << 30):
        prev = lib.mrpop_set_fused_edges(limit)
        try:
            out.append([t.cpu().numpy() for t in pkg.validate(scene, robots, a, b, 9, rule=rule, range_=1.1)])
        finally:
            lib.mrpop_set_fused_edges(prev)
    for other in out[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(out[0], other))
    assert scene.status() == 0
