"""The graph step's skin list where its cost depends on the scene: the order of the bodies, the
number of obstacles, the number of bodies. Results are compared with delta_sim_step bit for
bit; times only with those of a like scene, by ratios far from what was measured."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BODY_STATE = ("pos", "vel", "ang", "ref_ang", "rot")
STATE = BODY_STATE + ("x", "y", "z")
DRV_CERT = 8


def permuted(scene, order):
    """The scene with its bodies in another order."""
    n, off = scene["n_bodies"], scene["tri_offset"]
    count = np.diff(off)[order]
    tri = np.concatenate([np.arange(off[b], off[b + 1]) for b in order])
    vertex = (3 * tri[:, None] + np.arange(3)).reshape(-1)
    out = {"n_bodies": n, "tri_offset": np.concatenate([[0], np.cumsum(count)]).astype(np.int64),
           "tri_body": np.repeat(np.arange(n, dtype=np.int32), count)}
    for k, a in scene.items():
        if k in ("x", "y", "z", "rx", "ry", "rz"):
            out[k] = a[vertex].copy()
        elif k not in out:
            out[k] = np.asarray(a).reshape(n, -1)[order].reshape(-1).copy()
    return out


def layer(n, floor_first=False, spacing=0.03, height=0.0104):
    """n particles of 20 triangles in one layer, the skin's reach above a floor of two."""
    from delta_b200.scenarios import particle_cloud_scene

    side = int(np.ceil(np.sqrt(n)))
    k, h = np.arange(n), 0.6 * side * spacing + 1.0
    centres = np.stack([(k % side - side / 2) * spacing, np.full(n, height), (k // side - side / 2) * spacing], 1)
    floor = (np.array([[-h, 0, -h], [h, 0, -h], [h, 0, h], [-h, 0, h]], float), np.array([[0, 2, 1], [0, 3, 2]]))
    scene = particle_cloud_scene(centres, np.full(n, 0.01), np.full(n, 20), [floor], seed=3, perturb=(1.0, 1.0))
    return permuted(scene, np.concatenate([[n], np.arange(n)])) if floor_first else scene


def shelves(n, m, seed=0):
    """n particles of 20 triangles in a cube, and m small plates, most of them just under one."""
    from delta_b200.scenarios import particle_cloud_scene

    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1 / 3)))
    k = np.arange(n)
    centres = 0.03 * np.stack([k % side, k // (side * side), k // side % side], 1).astype(float)
    under = centres[rng.integers(0, n, m)] - [0.0, 0.0086, 0.0]
    under[rng.random(m) < 0.3] += 5.0
    plate = np.array([[-1, 0, -1], [1, 0, -1], [1, 0, 1], [-1, 0, 1]], float)
    plates = [(u + w * plate, np.array([[0, 2, 1], [0, 3, 2]])) for u, w in zip(under, rng.uniform(0.002, 0.05, m))]
    scene = particle_cloud_scene(centres, np.full(n, 0.01), np.full(n, 20), plates, seed=3, perturb=(1.0, 1.0))
    scene["eps"] = np.where(scene["obstacle"] != 0, rng.choice([1e-4, 2e-4, 3e-4], n + m), 1e-4)
    return scene


def moving(scene, velocity):
    """The scene with its particles at `velocity` (3,) or (n, 3)."""
    v = np.zeros((scene["n_bodies"], 3))
    v[scene["obstacle"] == 0] = velocity
    scene["vel"] = v.reshape(-1).copy()
    return scene


def same_run(ctx, scene, steps, dt=1e-5, driver=DRV_CERT):
    """`steps` graph steps in one call equal single steps; returns (skin statistics, contacts)."""
    from delta_b200.engine import Simulation, StepParams

    prm = StepParams.make(dt=dt, gravity=(0.0, 0.0, 0.0))
    runs = []
    for graph in (False, True):
        sim = Simulation(ctx, scene, driver)
        cps = sim.step(steps, prm, graph=graph)
        runs.append((cps, sim.state(), sim.counters()))
        skin = sim.skin_stats()
        sim.close()
    (c0, s0, n0), (c1, s1, n1) = runs
    assert np.array_equal(c0, c1)
    for k in STATE:
        assert np.array_equal(s0[k], s1[k]), k
    for k in ("steps", "body_pairs", "triangle_pairs", "solved"):
        assert n0[k] == n1[k], k
    return skin, int(c1.sum())


def rebuilding_step(ctx, scene, steps=48):
    """Seconds a step when every step rebuilds the list (the bodies cross half the skin)."""
    from delta_b200.engine import Simulation, StepParams

    prm = StepParams.make(dt=1e-5, gravity=(0.0, 0.0, 0.0))
    sim = Simulation(ctx, scene, DRV_CERT)
    sim.step(1, prm, graph=True)
    skin = sim.skin_stats()["skin"]
    sim.close()
    sim = Simulation(ctx, moving(dict(scene), [0.75 * skin / 1e-5, 0.0, 0.0]), DRV_CERT)
    start = {k: sim.dev.t[k].clone() for k in BODY_STATE}
    best = np.inf
    for _ in range(4):
        for k, v in start.items():
            sim.dev.t[k].copy_(v)
        t = time.perf_counter()
        sim.step(steps, prm, graph=True)
        best = min(best, time.perf_counter() - t)
    assert sim.skin_stats()["rebuilds"] >= 4 * (steps - 1)
    sim.close()
    return best / steps


@pytest.mark.parametrize("n", [513, 700, 5000])
def test_a_floor_as_the_first_body_is_ordered(ctx, n):
    """The floor's run of pairs (one first body) is longer than 512, and ordered by the bitmap."""
    rng = np.random.default_rng(n)
    scene = moving(layer(n, floor_first=True, height=0.0084), rng.uniform(-40.0, 40.0, (n, 3)) * (1.0, 0.05, 1.0))
    skin, contacts = same_run(ctx, scene, 12)
    assert skin["rebuilds"] >= 3 and contacts > 0, (skin, contacts)


def test_a_rebuild_costs_the_same_whichever_body_the_floor_is(ctx):
    """Counting ranked a run by its length squared: with the floor as the first body, 12,000
    particles on it, a step with a rebuild took 4 times that with the floor as the last."""
    assert rebuilding_step(ctx, layer(12000, floor_first=True)) < 2.0 * rebuilding_step(ctx, layer(12000))


@pytest.mark.parametrize("n,m", [(3, 25), (700, 24), (700, 25), (2000, 128), (5000, 129), (9000, 300)])
def test_many_obstacles_are_all_searched(ctx, n, m):
    """Obstacle boxes shared out between threads (fewer particles than threads: 5, 8 and 3
    groups) or not (9,000 particles), in stages of 128, with several margins among them."""
    rng = np.random.default_rng(n)
    scene = moving(shelves(n, m, seed=m), rng.uniform(-30.0, 30.0, (n, 3)))
    skin, contacts = same_run(ctx, scene, 12)
    assert skin["rebuilds"] >= 3 and contacts > 0, (skin, contacts)


def test_a_rebuild_with_many_obstacles_costs_little_more(ctx):
    """Every box was tested against every particle by one thread a particle: a step with a
    rebuild, 1,000 particles, took 5 times as long with 1,000 far obstacles as with none."""
    from delta_b200.scenarios import particle_cloud_scene

    def scene(m):
        k = np.arange(1000)
        centres = 0.03 * np.stack([k % 10, k // 100, k // 10 % 10], 1).astype(float)
        quad = np.array([[-9, 0, -9], [9, 0, -9], [9, 0, 9], [-9, 0, 9]], float)
        floors = [(quad - [0, 0.05 + 0.01 * i, 0], np.array([[0, 2, 1], [0, 3, 2]])) for i in range(m)]
        return particle_cloud_scene(centres, np.full(1000, 0.01), np.full(1000, 20), floors, seed=3)

    assert rebuilding_step(ctx, scene(1000)) < 2.5 * rebuilding_step(ctx, scene(1))


def kernels_of_a_step(ctx, scene):
    """Kernels in a replayed step without a rebuild."""
    from delta_b200 import lib
    from delta_b200.engine import Simulation, StepParams

    prm = StepParams.make(dt=1e-9, gravity=(0.0, 0.0, 0.0))
    sim = Simulation(ctx, scene, DRV_CERT)
    sim.step(2, prm, graph=True)
    counts = []
    for steps in (8, 24):
        before = lib().delta_launch_count(ctx.handle)
        sim.step(steps, prm, graph=True)
        counts.append(lib().delta_launch_count(ctx.handle) - before)
    sim.close()
    return (counts[1] - counts[0]) // 16


def test_the_route_changes_with_the_bodies_and_the_obstacles(ctx):
    """Up to 16,384 bodies and 2^23 bodies times obstacles one cluster keeps the list; beyond,
    the conditional node, whose check and filter are more kernels a step."""
    small = kernels_of_a_step(ctx, layer(16383))  # and the floor
    assert kernels_of_a_step(ctx, layer(16384)) > small
    assert kernels_of_a_step(ctx, shelves(8192, 1024)) == small
    assert kernels_of_a_step(ctx, shelves(8192, 1025)) > small


@pytest.mark.parametrize("kind", ["sparse", "long", "overflow"])
def test_the_conditional_node_equals_stepping(ctx, kind):
    """The skin list's other route, over rebuilds caused by motion inside graphs of eight steps
    (calls of 160 and more) and of one, with counters: more than 16,384 bodies and a short list (sorted and compacted
    by one CTA); a list above 32,768 keys (sorted and selected by the whole chip); a lattice
    squeezed until its list outgrows the capacity it got from the first, empty search."""
    from delta_b200.scenarios import particle_cloud_scene

    rng = np.random.default_rng(31)
    side, spacing, steps = {"sparse": (26, 0.05, 175), "long": (21, 0.0206, 175), "overflow": (26, 0.027, 175)}[kind]
    g = (np.arange(side) - (side - 1) / 2) * spacing
    cen = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    n = len(cen)
    if kind == "sparse":
        cen[1:400:2] = cen[0:400:2] + [0.018, 0.0, 0.0]  # 200 pairs that touch
    scene = particle_cloud_scene(cen, np.full(n, 0.0095 if kind == "overflow" else 0.01), np.full(n, 20), [], seed=9)
    scene = moving(scene, -200.0 * cen if kind == "overflow" else rng.uniform(-20.0, 20.0, (n, 3)))
    skin, contacts = same_run(ctx, scene, steps)
    assert contacts > 0
    if kind == "sparse":
        assert n > 16384 and skin["rebuilds"] >= 3 and skin["capacity"] <= 8192, skin
    elif kind == "long":
        assert skin["rebuilds"] >= 3 and skin["capacity"] > 32768, skin
    else:
        assert skin["capacity"] > 8192, skin  # grown past the first list's


def test_calls_on_both_sides_of_the_longer_graph_equal_stepping(ctx):
    """Eight steps are recorded as one graph once 64 steps are left or were replayed one by one:
    calls that fall short of it, reach it, and go on with it, contacts carried over."""
    from delta_b200.engine import Simulation, StepParams
    from delta_b200.scenarios import lattice_scene

    scene, prm, runs = lattice_scene(seed=8), StepParams.make(dt=1e-5), []
    for graph in (False, True):
        sim = Simulation(ctx, scene, DRV_CERT)
        cps = [sim.step(k, prm, graph=graph) for k in (20, 17, 19, 16, 1, 9, 80)]
        runs.append((np.concatenate(cps), sim.state(), sim.counters()))
        sim.close()
    (c0, s0, n0), (c1, s1, n1) = runs
    assert np.array_equal(c0, c1) and n0 == n1 and c0.sum() > 0
    for k in STATE:
        assert np.array_equal(s0[k], s1[k]), k


def test_short_calls_do_not_record_the_longer_graph(ctx):
    """A second call of eight steps replayed them as one graph, which it had to record first
    (with the conditional node three times the call)."""
    from delta_b200.engine import Simulation, StepParams

    scene, prm = layer(17000), StepParams.make(dt=1e-9, gravity=(0.0, 0.0, 0.0))
    second, later = [], []
    for _ in range(6):
        sim, times = Simulation(ctx, scene, DRV_CERT), []
        for _ in range(4):
            t = time.perf_counter()
            sim.step(8, prm, graph=True)
            times.append(time.perf_counter() - t)
        sim.close()
        second.append(times[1])
        later += times[2:]
    assert min(second) < 1.7 * min(later), (second, later)


@pytest.mark.parametrize("pairs", [8191, 8192, 16383, 16384, 40000])
def test_pair_counts_are_summed_at_any_capacity(ctx, pairs):
    """A step's contacts per pair are summed over the pair capacity and one: in one CTA, of one
    tile or two, up to 16,384 entries, beyond by cub."""
    from delta_b200.engine import Simulation, StepParams
    from delta_b200.scenarios import lattice_scene

    scene, prm, runs = lattice_scene(seed=9, nx=6, ny=4, nz=6), StepParams.make(dt=1e-5), []
    for graph in (False, True):
        sim = Simulation(ctx, scene, DRV_CERT)
        if graph:
            sim.set_graph_capacity(pairs, 4096)
        cps = sim.step(20, prm, graph=graph)
        runs.append((cps, sim.state(), sim.contacts()))
        sim.close()
    (c0, s0, k0), (c1, s1, k1) = runs
    assert np.array_equal(c0, c1) and c0.sum() > 0
    for k in STATE:
        assert np.array_equal(s0[k], s1[k]), k
    for k in ("depth", "master", "slave", "tri_a", "tri_b"):
        assert np.array_equal(k0[k], k1[k]), k
