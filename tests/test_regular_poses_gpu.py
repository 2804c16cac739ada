"""Edges whose joint values or bases are outside the range in which the kernels
use facts that hold for every pose (overlaps and screens of one arm's own
spheres), beside edges inside it: joint values far beyond a turn, edges that
cross the limit between two samples, and a base tens of metres out.  Verdicts
and first hits equal the oracle's with the device's __sinf/__cosf values
replayed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("arms,g,spread,shift", [(1, 33, 90.0, 0.0), (2, 32, 20.0, 0.0), (3, 17, 60.0, 0.0),
                                                 (4, 64, 25.0, 0.0), (4, 32, 0.0, 50.0), (5, 32, 15.0, 0.0)])
def test_poses_outside_the_regular_range(cuda, pkg, orc, split, arms, g, spread, shift):
    rng = np.random.default_rng(70 * arms + g)
    bases = pkg.workloads.bases_facing_centre(arms, 0.71).copy()
    bases[:, 0, 3] += np.float32(shift)
    q0, q1 = pkg.workloads.random_edges(rng, 192, arms, 1.5)
    far = rng.random(192) < 0.5
    q0[far] += rng.uniform(-spread, spread, (int(far.sum()), 7 * arms)).astype(np.float32)
    q1[far] = q0[far] + rng.normal(size=(int(far.sum()), 7 * arms)).astype(np.float32) * np.float32(0.05 * spread + 0.1)
    x = cuda.from_numpy(np.ascontiguousarray(orc.edge_samples(q0, q1, g, 0, 0.0), np.float32).ravel()).cuda()
    c, s = pkg.debug_trig(x)
    cuda.cuda.synchronize()
    trig = orc.TrigTable(x.cpu().numpy(), c.cpu().numpy(), s.cpu().numpy())
    sc = pkg.workloads.scene_config2(arms)
    sc.cuboids[:, 0] += np.float32(shift)
    scene, robots = pkg.Scene(sc), pkg.RobotSet(arms, bases)
    a, b = cuda.from_numpy(q0).cuda(), cuda.from_numpy(q1).cuda()
    both = pkg.CHECK_ENV | pkg.CHECK_SELF
    lib = pkg.library()
    prev = lib.mrpop_set_fused_edges(-1 if split else 0)
    try:
        for flags in (both, both | pkg.MODE_EXACT):
            v, f = pkg.validate(scene, robots, a, b, g, flags)
            ref = orc.validate(sc, bases, q0, q1, g, flags, trig=trig)
            assert np.array_equal(v.cpu().numpy(), ref["valid"])
            assert np.array_equal(f.cpu().numpy(), ref["first_hit"])
    finally:
        lib.mrpop_set_fused_edges(prev)
    assert scene.status() == 0
