"""B-spline and shortcut edges of thousands of segments.  Their samples add the
segment step once per finished segment, and the additions' rounding grows with
the segment number: at segment 4000 of these edges joints 2 to 4 (16 to 22 rad,
half an ulp of bias per addition) are 3.7e-3 rad from q0 + 4000 * step.  In each
edge one of the low intra-arm rows first touches, by 0.3 mm, seven or so
segments before the end, at the joint values with the rounding; without it the
sphere groups stay 0.3 to 1.2 mm out of reach.  Verdicts, first hits and segment
counts equal the oracle's with the device's __sinf/__cosf values replayed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEGMENTS = 4000
# joints 2..7 at the start, and joints 2..4 at the end (5..7 stay)
EDGES = [((-18.1606159, -19.828186, -21.3849163, -1.20533168, 0.870187938, -0.631214678),
          (-17.8515491, -19.5191193, -21.6939831)),
         ((-18.3362427, 18.1153011, -21.3734856, -1.27727211, 1.05369449, -1.28022337),
          (-18.0271759, 18.4243679, -21.6825523)),
         ((-19.9424782, -22.4589558, 16.8263912, -1.41192818, 1.02865541, -0.424615055),
          (-20.251545, -22.149889, 16.5173244)),
         ((-17.7108459, -18.4170628, 16.8591843, -1.60676408, 1.14298332, 2.14741111),
          (-17.4017792, -18.7261295, 16.5501175))]


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("arms,rule", [(1, 2), (1, 3), (2, 2), (3, 3)])
def test_late_hits_of_low_rows(cuda, pkg, orc, split, arms, rule):
    one0 = np.array([(0.3 * i, *a) for i, (a, _) in enumerate(EDGES)], np.float32)
    one1 = one0.copy()
    one1[:, 1:4] = [b for _, b in EDGES]
    # every arm makes the motion of another edge
    q0 = np.concatenate([np.roll(one0, a, axis=0) for a in range(arms)], axis=1)
    q1 = np.concatenate([np.roll(one1, a, axis=0) for a in range(arms)], axis=1)
    dist = np.sqrt(((q1[0].astype(float) - q0[0]) ** 2).sum())
    range_ = float((dist - (0.001 if rule == 3 else 0.0)) / (SEGMENTS - 0.5))
    bases = np.tile(np.eye(4, dtype=np.float32), (arms, 1, 1))
    bases[:, 0, 3] = 4.0 * np.arange(arms)
    sc = pkg.SceneArrays()
    x = cuda.from_numpy(np.ascontiguousarray(orc.edge_samples(q0, q1, 1, rule, range_), np.float32).ravel()).cuda()
    c, s = pkg.debug_trig(x)
    trig = orc.TrigTable(x.cpu().numpy(), c.cpu().numpy(), s.cpu().numpy())
    both = pkg.CHECK_ENV | pkg.CHECK_SELF
    scene, robots = pkg.Scene(sc), pkg.RobotSet(arms, bases)
    a, b = cuda.from_numpy(q0).cuda(), cuda.from_numpy(q1).cuda()
    lib = pkg.library()
    prev = lib.mrpop_set_fused_edges(-1 if split else 0)
    try:
        for flags in (both, both | pkg.MODE_EXACT):
            ref = orc.validate(sc, bases, q0, q1, 1, flags, rule=rule, range_=range_, trig=trig)
            assert np.all(ref["n_seg"] == SEGMENTS) and np.all(ref["first_hit"] > SEGMENTS - 20)
            v, f = pkg.validate(scene, robots, a, b, 1, flags, rule=rule, range_=range_)[:2]
            assert np.array_equal(v.cpu().numpy(), ref["valid"])
            assert np.array_equal(f.cpu().numpy(), ref["first_hit"])
    finally:
        lib.mrpop_set_fused_edges(prev)
    assert scene.status() == 0
