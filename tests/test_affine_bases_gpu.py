"""Arm bases that are not rigid transforms (larger, smaller, stretched, skewed
and mirrored frames) or far out: sphere centres follow the frame while radii do
not, so a bound that holds in a joint's own frame need not hold in the world.
Verdicts and first hits equal the oracle's with the device's __sinf/__cosf
values replayed, in the small-call kernels, the split kernels and a batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FRAMES = {
    "larger": np.diag([1.7, 1.7, 1.7]),
    "smaller": np.diag([0.55, 0.55, 0.55]),
    "stretched": np.diag([1.0, 1.45, 0.8]),
    "skewed": np.array([[1.0, 0.5, 0.0], [0.0, 1.0, 0.35], [0.0, 0.0, 1.0]]),
    "mirrored": np.diag([1.0, -1.0, 1.0]),
    "far": np.eye(3),
}


@pytest.mark.parametrize("form", ["small", "split", "one", "batch"])
@pytest.mark.parametrize("arms,g", [(1, 32), (2, 33), (3, 17), (4, 32), (5, 64)])
@pytest.mark.parametrize("frame", sorted(FRAMES))
def test_bases_that_are_not_rigid(cuda, pkg, orc, frame, arms, g, form):
    rng = np.random.default_rng(90 * arms + g)
    bases = pkg.workloads.bases_facing_centre(arms, 0.71).astype(np.float64)
    shift = 700.0 if frame == "far" else 0.0
    # every other arm only, so that arms inside and outside the rule meet
    for i in range(0, arms, 2):
        bases[i, :3, :3] = bases[i, :3, :3] @ FRAMES[frame]
    bases[:, 0, 3] += shift
    bases = bases.astype(np.float32)
    n = 64 if form == "batch" else 256
    q0, q1 = pkg.workloads.random_edges(rng, n, arms, 1.0)
    x = cuda.from_numpy(np.ascontiguousarray(orc.edge_samples(q0, q1, g, 0, 0.0), np.float32).ravel()).cuda()
    c, s = pkg.debug_trig(x)
    trig = orc.TrigTable(x.cpu().numpy(), c.cpu().numpy(), s.cpu().numpy())
    sc = pkg.workloads.scene_config2(arms)
    sc.cuboids[:, 0] += np.float32(shift)
    scene, robots = pkg.Scene(sc), pkg.RobotSet(arms, bases)
    a, b = cuda.from_numpy(q0).cuda(), cuda.from_numpy(q1).cuda()
    lib = pkg.library()
    # "one": split, the detailed phase of a middle-sized call; "split": a call above its limit, in copies
    copies = -(-(100000 // (arms * arms) + 1) // n) if form == "split" and arms > 1 else 1
    prev = lib.mrpop_set_fused_edges(0 if form == "small" else -1)
    try:
        for flags in (pkg.CHECK_SELF, pkg.CHECK_ENV | pkg.CHECK_SELF | pkg.MODE_EXACT):
            ref = orc.validate(sc, bases, q0, q1, g, flags, trig=trig)
            if form == "batch":
                batch = pkg.Batch([(scene, robots, a, b, g, flags, -1)])
                batch.run()
                cuda.cuda.synchronize()
                v, f = batch.valid[0], batch.first_hit[0]
            else:
                v, f = pkg.validate(scene, robots, a.repeat(copies, 1), b.repeat(copies, 1), g, flags)
            assert np.array_equal(v.cpu().numpy(), np.tile(ref["valid"], copies))
            assert np.array_equal(f.cpu().numpy(), np.tile(ref["first_hit"], copies))
    finally:
        lib.mrpop_set_fused_edges(prev)
    assert scene.status() == 0
