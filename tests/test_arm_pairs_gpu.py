"""Arm-vs-arm detailed tests where they can go wrong: arms so close that many
spheres of one reach the other (more than a lane's stash holds), first hits at
every sample, samples around the 32-sample slots, and arm pairs that never
meet.  Verdicts and first hits equal the oracle's with the device's
__sinf/__cosf values replayed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bases(pkg, arms, gap):
    return np.stack([pkg.workloads.yaw_base(gap * a, 0.0, 0.0, 0.7 * a) for a in range(arms)])


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("arms,gap,g", [(2, 0.12, 31), (2, 0.5, 64), (3, 0.3, 33), (4, 0.9, 32), (5, 0.3, 64),
                                        (5, 3.0, 48), (5, 0.7, 1)])
def test_arm_pairs_equal_the_oracle(cuda, pkg, orc, split, arms, gap, g):
    rng = np.random.default_rng(40 * arms + g)
    bases = _bases(pkg, arms, gap)
    q0, q1 = pkg.workloads.random_edges(rng, 160, arms, 3.0)
    x = cuda.from_numpy(np.ascontiguousarray(orc.edge_samples(q0, q1, g, 0, 0.0), np.float32).ravel()).cuda()
    c, s = pkg.debug_trig(x)
    cuda.cuda.synchronize()
    trig = orc.TrigTable(x.cpu().numpy(), c.cpu().numpy(), s.cpu().numpy())
    empty = pkg.SceneArrays()
    scene, robots = pkg.Scene(empty), pkg.RobotSet(arms, bases)
    a, b = cuda.from_numpy(q0).cuda(), cuda.from_numpy(q1).cuda()
    lib = pkg.library()
    prev = lib.mrpop_set_fused_edges(-1 if split else 0)
    try:
        for flags in (pkg.CHECK_SELF, pkg.CHECK_SELF | pkg.MODE_EXACT):
            v, f = pkg.validate(scene, robots, a, b, g, flags)
            ref = orc.validate(empty, bases, q0, q1, g, flags, trig=trig)
            assert np.array_equal(v.cpu().numpy(), ref["valid"])
            assert np.array_equal(f.cpu().numpy(), ref["first_hit"])
    finally:
        lib.mrpop_set_fused_edges(prev)
    assert scene.status() == 0
