"""Obstacle screens where they can go wrong: more obstacles than one or two
rounds of a warp, boxes whose axes are not orthonormal (their test is not a
distance, so no bound may use it), a capsule with an inconsistent 1/|v|^2,
obstacles the size of a fingertip and of the whole cell, and every class at
once.  Verdicts and first hits equal the oracle's with the device's
__sinf/__cosf values replayed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(pkg, rng, boxes, skewed, others):
    W = pkg.workloads

    def at():
        while True:
            c = rng.uniform((-1.1, -1.1, 0.0), (1.1, 1.1, 1.1))
            if np.hypot(abs(c[0]) - 0.5, abs(c[1]) - 0.5) > 0.35:
                return c

    cub = [W.box(at(), rng.uniform(-1, 1, 3), rng.uniform(0.004, 0.09, 3)) for _ in range(boxes)]
    for _ in range(skewed):
        b = W.box(at(), rng.uniform(-1, 1, 3), rng.uniform(0.02, 0.06, 3))
        b[3:12] += rng.normal(size=9).astype(np.float32) * np.float32(0.2)
        cub.append(b)
    kw = dict(cuboids=np.stack(cub))
    if others:
        caps = np.stack([W.capsule(at(), rng.uniform(-1, 1, 3), rng.uniform(0.01, 0.05), rng.uniform(0.05, 0.4))
                         for _ in range(others)])
        caps[0, 7] *= np.float32(0.5)
        kw.update(capsules=caps,
                  z_capsules=np.stack([W.capsule(at(), (0, 0, 0), 0.03, rng.uniform(0.05, 0.4)) for _ in range(others)]),
                  z_cuboids=np.stack([W.box(at(), (0, 0, rng.uniform(-3, 3)), rng.uniform(0.01, 0.08, 3))
                                      for _ in range(others)]),
                  spheres=np.stack([np.array([*at(), rng.uniform(0.005, 0.08)], np.float32) for _ in range(others)]))
    return pkg.SceneArrays(**kw)


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("arms,g,boxes,skewed,others", [(1, 32, 31, 0, 0), (1, 64, 20, 13, 0), (2, 32, 9, 4, 11),
                                                        (4, 33, 65, 0, 3), (4, 16, 12, 12, 12), (3, 1, 40, 2, 2)])
def test_obstacle_screens(cuda, pkg, orc, split, arms, g, boxes, skewed, others):
    rng = np.random.default_rng(boxes * 100 + g)
    sc = _scene(pkg, rng, boxes, skewed, others)
    bases = pkg.workloads.bases_config2()[:arms]
    q0, q1 = pkg.workloads.random_edges(rng, 256, arms, 2.0)
    x = cuda.from_numpy(np.ascontiguousarray(orc.edge_samples(q0, q1, g, 0, 0.0), np.float32).ravel()).cuda()
    c, s = pkg.debug_trig(x)
    cuda.cuda.synchronize()
    trig = orc.TrigTable(x.cpu().numpy(), c.cpu().numpy(), s.cpu().numpy())
    scene, robots = pkg.Scene(sc), pkg.RobotSet(arms, bases)
    a, b = cuda.from_numpy(q0).cuda(), cuda.from_numpy(q1).cuda()
    both = pkg.CHECK_ENV | pkg.CHECK_SELF
    lib = pkg.library()
    prev = lib.mrpop_set_fused_edges(-1 if split else 0)
    try:
        for flags in (both, pkg.CHECK_ENV, both | pkg.MODE_EXACT):
            v, f = pkg.validate(scene, robots, a, b, g, flags)
            ref = orc.validate(sc, bases, q0, q1, g, flags, trig=trig)
            assert np.array_equal(v.cpu().numpy(), ref["valid"])
            assert np.array_equal(f.cpu().numpy(), ref["first_hit"])
    finally:
        lib.mrpop_set_fused_edges(prev)
    assert scene.status() == 0
