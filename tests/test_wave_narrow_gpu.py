"""Split service waves on both sides of the size up to which the narrow phase is
one kernel (100000 / arms^2 edges, twice that for segmented steps): a session's
step gives the direct call's verdicts and first hits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rule,g,n", [(0, 33, 3999), (0, 32, 4001), (3, 17, 7999), (1, 64, 8001)])
def test_steps_around_the_limit(cuda, pkg, rule, g, n):
    arms = 5
    W = pkg.workloads
    bases = W.bases_config3()
    q0, q1 = W.random_edges(np.random.default_rng(n), n, arms, 2.0)
    scene, robots = pkg.Scene(W.scene_config3(4)), pkg.RobotSet(arms, bases)
    flags, range_ = pkg.CHECK_ENV | pkg.CHECK_SELF, 1.3 if rule else 0.0
    server = pkg.Server(budget_bytes=256 << 20, streams=1, fused_edges=-1)
    sess = server.session(arms, n, 64)
    v, f = sess.validate(scene, robots, q0, q1, g, flags, -1, rule, range_)
    v2, f2 = sess.validate(scene, robots, q0, q1, g, flags, -1, rule, range_)
    sess.close()
    server.close()
    a, b = cuda.from_numpy(q0).cuda(), cuda.from_numpy(q1).cuda()
    out = pkg.validate(scene, robots, a, b, g, flags, -1, rule, range_)
    cuda.cuda.synchronize()
    assert 0 < int(v.sum()) < n
    for x, y in ((v, f), (v2, f2)):
        assert np.array_equal(x, out[0].cpu().numpy())
        assert np.array_equal(y, out[1].cpu().numpy())
    assert scene.status() == 0


@pytest.mark.parametrize("arms,rule,limit", [(1, 0, 4096), (2, 0, 4096), (3, 0, 2048), (5, 0, 2048), (4, 2, 4096),
                                             (5, 3, 3072)])
def test_default_limit_of_fused_groups(cuda, pkg, arms, rule, limit):
    """A wave of one fused group is one launch; above the limit, or above one set, it is several."""
    W = pkg.workloads
    bases = W.bases_facing_centre(arms, 0.71)
    q0, q1 = W.random_edges(np.random.default_rng(limit), limit + 1, arms, 2.0)
    scene, robots = pkg.Scene(W.scene_config2(3)), pkg.RobotSet(arms, bases)
    for setting in (0, 1000):
        server = pkg.Server(budget_bytes=256 << 20, streams=1, fused_edges=setting)
        sess = server.session(arms, limit + 1, 8)
        bound, launches = setting or limit, []
        for n in (bound, bound + 1):
            before = server.stats()["kernel_launches"]
            sess.validate(scene, robots, q0[:n], q1[:n], 8, rule=rule, range_=1.0 if rule else 0.0)
            launches.append(server.stats()["kernel_launches"] - before)
        sess.close()
        server.close()
        assert launches[0] == 1 and launches[1] > 1
