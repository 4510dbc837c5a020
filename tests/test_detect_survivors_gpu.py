"""Detections with many survivors of the box culling: every pair of long thin triangles that
cross the same space has overlapping boxes, and few of them touch."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x", "normal", "depth", "P", "Q", "eps_total", "master", "slave", "tri_a", "tri_b")


def needles(triangles, seed):
    """Vertices (3 * triangles, 3) of thin triangles, each across the unit cube."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.0, 0.2, (triangles, 3))
    b = rng.uniform(0.8, 1.0, (triangles, 3))
    flip = rng.random((triangles, 3)) < 0.5  # along the four diagonals
    a, b = np.where(flip, b, a), np.where(flip, a, b)
    return np.stack([a, b, b + rng.uniform(-0.01, 0.01, (triangles, 3))], 1).reshape(-1, 3)


def bodies(sizes, seed=0, eps=5e-6):
    from delta_b200 import detection

    xyz = np.concatenate([needles(n, seed + k) for k, n in enumerate(sizes)])
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = len(sizes)
    return detection.Meshes(off, *(xyz[:, k].copy() for k in range(3)), np.full(n, eps), np.zeros(n, np.uint8))


def detect(ctx, driver, meshes, pairs, contacts):
    import torch

    from delta_b200 import lib

    pa, pb = (torch.tensor(p, dtype=torch.int32).cuda() for p in zip(*pairs))
    count = ctypes.c_int64(0)
    launches = lib().delta_launch_count(ctx.handle)
    status = lib().delta_detect(ctx.handle, driver, 0, ctypes.byref(meshes.struct()), pa.data_ptr(), pb.data_ptr(),
                                len(pairs), ctypes.byref(contacts.struct()), ctypes.byref(count), None)
    assert status == 0, status
    rows = contacts.to_numpy(count.value)
    return rows, lib().delta_launch_count(ctx.handle) - launches


@pytest.mark.parametrize("name", ["bf", "bf_cert", "bf_culled", "learned"])
def test_a_long_survivor_list_is_kept_from_call_to_call(name):
    """160,801 survivors do not fit a new context's list of 65,536: the first call culls twice,
    the later ones launch each kernel once, and all return the contacts of a context whose list
    was long enough from the start."""
    from delta_b200 import detection
    from delta_b200.narrowphase import Context

    driver = {"bf": detection.DRV_BF, "bf_cert": detection.DRV_BF_CERT, "bf_culled": detection.DRV_BF_CULLED,
              "learned": detection.DRV_LEARNED}[name]
    sizes, pairs = [401] * 6, [(k, k + 1) for k in range(5)]  # 804,005 triangle pairs
    m = bodies(sizes)
    ctx = Context(0)
    runs = [detect(ctx, driver, m, pairs, detection.Contacts(4096)) for _ in range(3)]
    ctx.close()
    long = Context(0)
    want, least = detect(long, driver, m, pairs, detection.Contacts(1 << 17))
    long.close()
    assert 0 < len(want) <= 4096
    for rows, _ in runs:
        assert len(rows) == len(want)
        for f in FIELDS:
            assert np.array_equal(rows[f], want[f]), f
    assert runs[0][1] > least and [n for _, n in runs[1:]] == [least, least]


@pytest.mark.parametrize("sizes,pairs", [
    ([1, 1], [(0, 1)]),                                          # one slice
    ([33, 600, 129, 2000], [(0, 1), (1, 0), (1, 2), (2, 3), (3, 1)]),  # slices with remainders, empty ones
    ([1500, 1499], [(0, 1)]),
    ([6000, 2], [(0, 1)]),                                       # second bodies too small to cut
    ([60000, 2], [(0, 1)]),                                      # uneven: every triangle pair is solved
    ([30] * 40 + [2500, 2500], [(k, k + 1) for k in range(39)] * 20 + [(40, 41)]),  # one large pair among small ones
], ids=["one", "mixed", "pair", "flat", "flat_uneven", "uneven"])
def test_bf_in_slices_equals_the_unsliced_culling(ctx, sizes, pairs):
    """bf() culls slices of the second bodies, or solves every triangle pair where one large
    body pair would hold up one block: the contacts of the culling with one block to a pair,
    bit for bit."""
    from delta_b200 import detection

    m = bodies(sizes, seed=7, eps=2e-4 if max(sizes) < 100 else 2e-5)
    got, _ = detect(ctx, detection.DRV_BF, m, pairs, detection.Contacts(1 << 17))
    want, _ = detect(ctx, detection.DRV_BF_CULLED, m, pairs, detection.Contacts(1 << 17))
    assert len(got) == len(want) and (len(want) > 0 or sum(sizes) < 10)
    for f in FIELDS:
        assert np.array_equal(got[f], want[f]), f


def test_bf_on_two_large_bodies_uses_the_whole_chip(ctx):
    """Two spheres of 5,120 triangles, one half inside the other: bf() took one block of the
    culling 16 ms; in slices, or with every triangle pair solved, it takes less than half."""
    import time

    from delta_b200 import detection
    from delta_b200.scenarios import sphere_mesh

    V, F = sphere_mesh(5120, None, 0.5)
    xyz = np.concatenate([V[F].reshape(-1, 3), (V + [0.3, 0.013, 0.007])[F].reshape(-1, 3)])
    m = detection.Meshes(np.array([0, 5120, 10240]), *(xyz[:, k].copy() for k in range(3)), np.full(2, 1e-4),
                         np.zeros(2, np.uint8))
    least = {}
    for driver in (detection.DRV_BF, detection.DRV_BF_CULLED):
        contacts, times = detection.Contacts(4096), []
        for _ in range(4):
            t = time.perf_counter()
            detect(ctx, driver, m, [(0, 1)], contacts)
            times.append(time.perf_counter() - t)
        least[driver] = min(times)
    assert least[detection.DRV_BF] < 0.5 * least[detection.DRV_BF_CULLED], least


def test_bf_bounds_its_survivor_list():
    """bf() needs no memory for the triangle pairs that it solves one by one, so the list of its
    culling is bounded: four pairs with 77 million survivors (0.6 GB) are solved without one.
    The contacts are those of the driver that lists them all."""
    import torch

    from delta_b200 import detection
    from delta_b200.narrowphase import Context

    m = bodies([4400] * 5, seed=11, eps=1e-7)
    pairs = [(k, k + 1) for k in range(4)]
    rows = {}
    for driver in (detection.DRV_BF, detection.DRV_BF_CULLED):
        ctx, contacts = Context(0), detection.Contacts(1 << 17)
        free = torch.cuda.mem_get_info()[0]
        rows[driver], _ = detect(ctx, driver, m, pairs, contacts)
        used = free - torch.cuda.mem_get_info()[0]
        ctx.close()
        if driver == detection.DRV_BF:
            assert used < 200 << 20, used
    got, want = rows.values()
    assert len(got) == len(want) > 0
    for f in FIELDS:
        assert np.array_equal(got[f], want[f]), f
