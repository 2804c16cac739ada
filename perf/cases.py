"""Timed cases of the edge validator, the sphere placement and the planner.

A case is one call (or one planner solve) that a program using this library
makes, through the Python binding of the C ABI: `validate` on CUDA tensors,
`Workspace.validate` on page-locked host arrays, a `Batch` of planning
instances, `fk_spheres`, and `drrt.solve`.  Scenes, arm layouts and edges come
from the package's seeded workload generators.

Kinds of case and their fields:
  edges  arms, n, g, rule, range, flags ("both", "self", "env", "exact"),
         scene, length, single (check arm arms // 2 alone), start ("any": edges
         start anywhere within the joint limits, as in the benchmark's batches;
         "free": at one of a few thousand collision-free nodes, as a
         planner's do)
  host   the same, from page-locked host buffers
  batch  instances, scale: that many planning instances of 1 to 5 arms
  fk     n configurations of one arm, detailed or broad-phase spheres
  solve  arms, attempts, g, range: one planner solve with the served stream's
         budget
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

RULES = {"plain": 0, "connect": 1, "bspline": 2, "shortcut": 3}


def listed():
    return [
        # One iteration of the planner's tree growth: its 300 extension
        # attempts, composite self check only, 64 samples each.  The call a
        # solve makes most often; latency is all that counts.
        dict(name="extend_5arm_300x64", kind="edges", arms=5, n=300, g=64, rule="plain", range=0.0, flags="self",
             scene="shelf", length=2.0, single=False, start="free"),
        # The same iteration's new nodes towards the other tree: connect
        # segments of `range`, scene and arms.
        dict(name="connect_4arm_300x64", kind="edges", arms=4, n=300, g=64, rule="connect", range=2.0, flags="both",
             scene="bins", length=6.0, single=False, start="free"),
        # A roadmap round's new samples of one arm, checked as nodes.
        dict(name="nodes_1arm_1840x1", kind="edges", arms=4, n=1840, g=1, rule="plain", range=0.0, flags="both",
             scene="bins", length=0.0, single=True, start="any"),
        # One arm among boxes and capsules: an ordinary single-robot batch.
        dict(name="single_1arm_4096x32", kind="edges", arms=1, n=4096, g=32, rule="plain", range=0.0, flags="both",
             scene="clutter", length=1.0, single=True, start="any"),
        # A roadmap round's candidate edges of one arm of a four-arm cell.
        dict(name="roadmap_1arm_30011x32", kind="edges", arms=4, n=30011, g=32, rule="plain", range=0.0, flags="both",
             scene="bins", length=1.5, single=True, start="free"),
        # Path smoothing from host code: three arms, candidate corners as
        # B-spline segments, every flagged sample checked, all obstacle classes.
        dict(name="host_bspline_3arm_2777x24", kind="host", arms=3, n=2777, g=24, rule="bspline", range=0.7,
             flags="exact", scene="mixed", length=3.0, single=False, start="free"),
        # Four arms around a bin-picking table: the benchmark's batch.
        dict(name="quad_4arm_65536x32", kind="edges", arms=4, n=65536, g=32, rule="plain", range=0.0, flags="both",
             scene="bins", length=1.5, single=False, start="any"),
        # Five arms at a shelf, 64 samples: the largest plain batch.
        dict(name="shelf_5arm_262144x64", kind="edges", arms=5, n=262144, g=64, rule="plain", range=0.0,
             flags="both", scene="shelf", length=1.5, single=False, start="any"),
        # Shortcut candidates of many paths at once: long edges, several
        # segments each, early exit at the first collision.
        dict(name="shortcut_5arm_65536x64", kind="edges", arms=5, n=65536, g=64, rule="shortcut", range=2.0,
             flags="both", scene="shelf", length=5.0, single=False, start="free"),
        # Uneven planning instances of 1 to 5 arms validated as one batch.
        dict(name="batch_128_instances", kind="batch", instances=128, scale=1.0),
        # Sphere centres of a roadmap's worth of configurations, for display
        # or for a caller's own distance queries.
        dict(name="fk_detailed_100000", kind="fk", n=100000, detailed=True),
        # A whole planner solve (roadmaps, tree growth, simplification).
        dict(name="solve_4arm", kind="solve", arms=4, attempts=64, g=32, range=1.5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["edges"] * 6 + ["host"] * 2 + ["batch", "fk", "solve"])
    if kind == "batch":
        return dict(kind="batch", instances=rng.randint(9, 128), scale=round(rng.uniform(0.05, 0.9), 3))
    if kind == "fk":
        return dict(kind="fk", n=_log_int(rng, 30, 400000), detailed=rng.random() < 0.5)
    if kind == "solve":
        return dict(kind="solve", arms=rng.randint(2, 4), attempts=rng.randint(32, 96), g=rng.randint(16, 48),
                    range=round(rng.uniform(1.0, 1.6), 3))
    arms = rng.randint(1, 5)
    single = arms == 1 or rng.random() < 0.25
    g = rng.choice([1, 2, 8, 16, 17, 31, 32, 33, 48, 63, 64, rng.randint(3, 64)])
    rule = rng.choice(["plain", "plain", "connect", "bspline", "shortcut"])
    # arm-samples of a segment, at most half those of the largest listed case
    most = 40e6 / (g * (1 if single else arms) * (1 if rule == "plain" else 4))
    # (fewer edges than the lower end are often all free, whatever the seed)
    n = _log_int(rng, 48, max(96, min(300000 if kind == "edges" else 40000, most)))
    return dict(kind=kind, arms=arms, n=n, g=g, rule=rule,
                range=0.0 if rule == "plain" else round(rng.uniform(0.5, 2.5), 3),
                flags=rng.choice(["both", "both", "exact"] + ([] if single else ["both", "self", "env"])),
                scene=rng.choice(["mixed", {1: "clutter", 5: "shelf"}.get(arms, "bins")]),
                length=round(rng.uniform(0.2, 2.0) if rule == "plain" else rng.uniform(0.5, 6.0), 3), single=single,
                start=rng.choice(["any", "free"]))


def _scene(pkg, kind, seed, bases):
    """The obstacles of a case: a generator of the package, or a cell with
    every class of obstacle the library tests, clear of the arms' bases."""
    w = pkg.workloads
    if kind == "clutter":
        return w.scene_config1(seed)
    if kind == "bins":
        return w.scene_config2(seed)
    if kind == "shelf":
        return w.scene_config3(seed)
    rng = np.random.default_rng(7000 + seed)

    def at():
        while True:
            c = rng.uniform((-1.3, -1.3, 0.0), (1.3, 1.3, 1.2))
            if min(math.hypot(*(c[:2] - b[:2, 3])) for b in bases) > 0.45:
                return c

    def caps(n, tilt):
        return np.stack([w.capsule(at(), rng.uniform(-tilt, tilt, 3), rng.uniform(0.02, 0.06), rng.uniform(0.1, 0.3))
                         for _ in range(n)])

    def boxes(n, tilt):
        return np.stack([w.box(at(), (*rng.uniform(-tilt, tilt, 2), rng.uniform(-3.0, 3.0)),
                               rng.uniform(0.02, 0.1, 3)) for _ in range(n)])

    spheres = np.stack([np.array([*at(), rng.uniform(0.02, 0.08)], np.float32) for _ in range(9)])
    return pkg.SceneArrays(spheres=spheres, capsules=caps(7, 1.0), z_capsules=caps(5, 0.0), cuboids=boxes(11, 1.0),
                           z_cuboids=boxes(6, 0.0))


def _bases(pkg, arms):
    w = pkg.workloads
    return w.bases_config2() if arms == 4 else w.bases_config3() if arms == 5 else w.bases_facing_centre(arms, 0.71)


def _flags(pkg, name):
    both = pkg.CHECK_ENV | pkg.CHECK_SELF
    return {"both": both, "self": pkg.CHECK_SELF, "env": pkg.CHECK_ENV, "exact": both | pkg.MODE_EXACT}[name]


def _instances(case):
    """Arms, edges, samples an edge and kind of scene of a batch's instances:
    lognormal edge counts, 1 to 5 arms, one arm among clutter, more at a table
    or in a mixed cell."""
    rng = np.random.default_rng(4400)
    return [(int(rng.integers(1, 6)), max(1, round(case["scale"] * float(rng.lognormal(math.log(2000.0), 1.0)))),
             int(rng.choice([16, 32, 64])), rng.random() < 0.5) for _ in range(case["instances"])]


def _configs(n, seed):
    """n configurations of one arm within the joint limits, as numpy float32."""
    w = load_package().workloads
    return w.random_configs(np.random.default_rng(6000 + seed), n, 1)


def _edges(pkg, scene, robots, arm, case, seed):
    """A case's edges as numpy float32: [n][7 * arms checked] each."""
    w = pkg.workloads
    rng = np.random.default_rng(5500 + seed)
    arms = 1 if arm >= 0 else robots.n_arms
    q0, q1 = w.random_edges(rng, case["n"], arms, case["length"])
    if case["start"] == "any":
        return q0, q1
    nodes = w.random_configs(rng, 16384, arms)
    t = torch.from_numpy(nodes).cuda()
    nodes = nodes[pkg.validate(scene, robots, t, t, 1, _flags(pkg, "both"), arm)[0].cpu().numpy() != 0]
    if len(nodes) == 0:
        return q0, q1
    start = nodes[rng.integers(0, len(nodes), case["n"])]
    lo, hi = np.tile(w.PANDA_LO, arms), np.tile(w.PANDA_HI, arms)
    return start, np.clip(start + (q1 - q0), lo, hi).astype(np.float32)


def prepare(case, seed):
    pkg = load_package()
    w = pkg.workloads
    kind = case["kind"]
    if kind == "batch":
        items, keep = [], []
        sizes, rng = _instances(case), np.random.default_rng(5700 + seed)
        for arms, n, g, mixed in sizes:
            bases = w.bases_facing_centre(arms, 0.71)
            name = "clutter" if arms == 1 else "mixed" if mixed else "bins"
            scene = pkg.Scene(_scene(pkg, name, int(rng.integers(1 << 30)), bases))
            robots = pkg.RobotSet(arms, bases)
            q0, q1 = (torch.from_numpy(q).cuda() for q in w.random_edges(rng, n, arms, 1.5))
            keep.append((scene, robots, q0, q1))
            items.append((scene, robots, q0, q1, g, _flags(pkg, "both"), -1))
        n = sum(m for _, m, _, _ in sizes)
        valid = torch.empty(n, dtype=torch.uint8, device="cuda")
        first = torch.empty(n, dtype=torch.int32, device="cuda")
        at = 0
        for i, it in enumerate(items):
            m = int(it[2].shape[0])
            items[i] = (*it, valid[at:at + m], first[at:at + m])
            at += m
        batch = pkg.Batch(items)
        batch.capture()
        return dict(kind=kind, batch=batch, valid=valid, first=first, keep=keep)
    if kind == "fk":
        return dict(kind=kind, pkg=pkg, robots=pkg.RobotSet(4, w.bases_config2()),
                    q=torch.from_numpy(_configs(case["n"], seed)).cuda(), detailed=case["detailed"])
    if kind == "solve":
        def free(scene, bases, q):
            t = torch.from_numpy(q).cuda()
            return pkg.validate(pkg.Scene(scene), pkg.RobotSet(len(bases), bases), t, t, 1)[0].cpu().numpy() != 0

        query = pkg.planner.make_queries(1, seed, free, arms_range=(case["arms"], case["arms"]))[0]
        settings = pkg.serving.served_drrt_settings(blocking_wait=0, num_new_configs=case["attempts"],
                                                    granularity=case["g"], range=case["range"])
        settings.seed = query.seed
        return dict(kind=kind, pkg=pkg, scene=pkg.Scene(query.scene), robots=pkg.RobotSet(query.arms, query.bases),
                    start=query.start, goal=query.goal, settings=settings)
    arms = case["arms"]
    bases = _bases(pkg, arms)
    scene, robots = pkg.Scene(_scene(pkg, case["scene"], seed, bases)), pkg.RobotSet(arms, bases)
    arm = arms // 2 if case["single"] else -1
    q0, q1 = _edges(pkg, scene, robots, arm, case, seed)
    st = dict(kind=kind, pkg=pkg, scene=scene, robots=robots, g=case["g"], flags=_flags(pkg, case["flags"]), arm=arm,
              rule=RULES[case["rule"]], range_=case["range"])
    if kind == "host":
        n = case["n"]
        pinned = dict(q0=torch.from_numpy(q0).pin_memory(), q1=torch.from_numpy(q1).pin_memory(),
                      valid=torch.empty(n, dtype=torch.uint8).pin_memory(),
                      first=torch.empty(n, dtype=torch.int32).pin_memory())
        st.update({k: t.numpy() for k, t in pinned.items()}, pinned=pinned, ws=pkg.Workspace())
    else:
        st.update(q0=torch.from_numpy(q0).cuda(), q1=torch.from_numpy(q1).cuda())
    return st


def run(s):
    kind = s["kind"]
    if kind == "edges":
        return s["pkg"].validate(s["scene"], s["robots"], s["q0"], s["q1"], s["g"], s["flags"], s["arm"], s["rule"],
                                 s["range_"])
    if kind == "host":
        return s["ws"].validate(s["scene"], s["robots"], s["q0"], s["q1"], s["g"], s["flags"], s["arm"], s["rule"],
                                s["range_"], s["valid"], s["first"])
    if kind == "batch":
        s["batch"].launch()
        return s["valid"], s["first"]
    if kind == "fk":
        return s["pkg"].fk_spheres(s["robots"], 1, s["q"], s["detailed"])
    r = s["pkg"].drrt.solve(s["scene"], s["robots"], s["start"], s["goal"], s["settings"])
    t = r.stats
    counters = [int(r.solved), r.iters, t["iterations"], t["launches"], t["validate_calls"], t["edges_validated"],
                t["start_tree_size"], t["goal_tree_size"], *t["roadmap_nodes"], *t["roadmap_edges"]]
    counters += [len(r.path), len(r.solutions)]
    path, costs = np.zeros((512, len(s["start"])), np.float32), np.zeros(8, np.float32)
    path[:len(r.path)] = r.path
    costs[:len(r.solutions)] = [x.cost for x in r.solutions]
    return {"path": path, "costs": costs, "counters": np.array(counters, np.int64)}


# Flops of placing one arm's 11 broad-phase spheres: 7 joint composes of 81
# and 11 placements of 18 (FMA = 2).  Collision tests can be culled; these
# cannot.
_FK_FLOPS = 7 * 81 + 11 * 18


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = _instances(case)
        return {"bytes": sum(n * (2 * 28 * a + 5) for a, n, _, _ in sizes),
                "flops": sum(n * g * a * _FK_FLOPS for a, n, g, _ in sizes)}
    if kind == "fk":
        spheres = 59 if case["detailed"] else 11
        return {"bytes": case["n"] * 4 * (7 + 3 * spheres), "flops": case["n"] * (7 * 81 + spheres * 18)}
    if kind == "solve":
        # roadmaps: at least one round of 4 blocks of 230 samples an arm, as nodes
        n = 920 * case["arms"]
        return {"bytes": n * (28 + 5), "flops": n * _FK_FLOPS}
    arms = 1 if case["single"] else case["arms"]
    # segmented rules: at least every edge's first segment
    return {"bytes": case["n"] * (2 * 28 * arms + 5 + (4 if kind == "edges" and case["rule"] != "plain" else 0)),
            "flops": case["n"] * case["g"] * arms * _FK_FLOPS}


# The arm's sphere model: centres in the frame of their joint (0 = base).
_APPROX = [(0, 0, 0, .05), (1, -.001, -.039, -.085), (2, 0, -.085, .04), (3, .039, .028, -.052),
           (4, -.042, .049, .029), (5, -.001, .037, -.11), (6, .042, .014, 0), (7, .015, .015, .075),
           (7, 0, 0, .129), (7, .054447, .054447, .1984), (7, -.054447, -.054447, .1984)]
_DETAILED = [(0, 0, 0, .05), (1, 0, -.08, 0), (1, 0, -.03, 0), (1, 0, 0, -.12), (1, 0, 0, -.17), (2, 0, 0, .03),
             (2, 0, 0, .08), (2, 0, -.12, 0), (2, 0, -.17, 0), (3, 0, 0, -.1), (3, 0, 0, -.06), (3, .08, .06, 0),
             (3, .08, .02, 0), (4, -.08, .095, 0), (4, 0, 0, .02), (4, 0, 0, .06), (4, -.08, .06, 0), (5, 0, .055, 0),
             (5, 0, .075, 0), (5, 0, 0, -.22), (5, 0, .05, -.18)]
_DETAILED += [(5, x, y, z) for x in (.01, -.01) for y, z in ((.08, -.14), (.085, -.11), (.09, -.08), (.095, -.05))]
_DETAILED += [(6, 0, 0, 0), (6, .08, -.01, 0), (6, .08, .035, 0), (7, 0, 0, .07), (7, .02, .04, .08),
              (7, .04, .02, .08), (7, .04, .06, .085), (7, .06, .04, .085)]
_DETAILED += [(7, d, d, z) for z in (.117, .137, .157) for d in (-.053033, -.03182, -.010607, .010607, .03182, .053033)]
_DETAILED += [(7, .056569, .056569, .1874), (7, .051619, .051619, .2094), (7, -.056569, -.056569, .1874),
              (7, -.051619, -.051619, .2094)]
# Fixed transform before each joint: rotation about x by this many quarter
# turns, and translation.
_JOINTS = [(0, (0, 0, .333)), (-1, (0, 0, 0)), (1, (0, -.316, 0)), (1, (.0825, 0, 0)), (-1, (-.0825, .384, 0)),
           (1, (0, 0, 0)), (1, (.088, 0, 0))]


def exact(case, seed):
    if case["kind"] != "fk":
        return None  # verdicts and counters are whole numbers; a path follows from them
    q = _configs(case["n"], seed).astype(np.float64)
    at = math.atan2(.5, .5)  # arm 1 of the four: corner (-0.5, -0.5), facing the centre
    frame = np.array([[np.float32(math.cos(at)), -np.float32(math.sin(at)), 0, -.5],
                      [np.float32(math.sin(at)), np.float32(math.cos(at)), 0, -.5], [0, 0, 1, 0], [0, 0, 0, 1]])
    frames = [np.broadcast_to(frame, (len(q), 4, 4))]
    for j, (turn, shift) in enumerate(_JOINTS):
        c, s = np.cos(q[:, j]), np.sin(q[:, j])
        step = np.zeros((len(q), 4, 4))
        step[:, 0, 0], step[:, 0, 1] = c, -s
        if turn:
            step[:, 2, 0], step[:, 2, 1], step[:, 1, 2] = turn * s, turn * c, -turn
        else:
            step[:, 1, 0], step[:, 1, 1], step[:, 2, 2] = s, c, 1
        step[:, :3, 3] = np.float32(shift)
        step[:, 3, 3] = 1
        frames.append(frames[-1] @ step)
    out = []
    for j, x, y, z in _DETAILED if case["detailed"] else _APPROX:
        out.append(frames[j][:, :3, :] @ np.array([np.float32(x), np.float32(y), np.float32(z), 1.0]))
    return np.stack(out, axis=1)
