"""Small composite calls around the sizes at which the arm-per-warp kernel
changes from two warps per arm to one, and to the pair and one-warp kernels:
plain and connect edges give the split pipeline's results (which the parity
suite compares with the oracle), and the oracle's on a subset."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arms", [3, 4, 5])
@pytest.mark.parametrize("g", [32, 33, 64])
def test_small_composite_calls(cuda, pkg, arms, g):
    W = pkg.workloads
    bases = W.bases_config2() if arms == 4 else W.bases_facing_centre(arms, 0.71)
    scene, robots = pkg.Scene(W.scene_config2(arms)), pkg.RobotSet(arms, bases)
    rng = np.random.default_rng(900 + arms)
    q0, q1 = W.random_edges(rng, 609, arms, 2.5)
    a, b = cuda.from_numpy(q0).cuda(), cuda.from_numpy(q1).cuda()
    lib = pkg.library()
    for rule, range_ in ((0, 0.0), (1, 0.8)):
        prev = lib.mrpop_set_fused_edges(-1)
        try:
            ref = [t.cpu().numpy() for t in pkg.validate(scene, robots, a, b, g, rule=rule, range_=range_)]
        finally:
            lib.mrpop_set_fused_edges(prev)
        for n in (1, 2, 151, 152, 153, 303, 304, 305, 456, 457, 608, 609):
            got = pkg.validate(scene, robots, a[:n].contiguous(), b[:n].contiguous(), g, rule=rule, range_=range_)
            assert all(np.array_equal(x.cpu().numpy(), y[:n]) for x, y in zip(got, ref)), (rule, n)
    assert scene.status() == 0
