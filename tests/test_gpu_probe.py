"""GPU tests of the probed check (a first pass over a voxel grid of each
environment, the undecided pairs walked from a queue): bit for bit the verdicts
of the one-pass check, at the edges of its batches, lists, grids and queue."""
import numpy as np
import pytest

from bcc import EnvSet, workload
from bcc.workload import make_cuboids, make_spheres
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def both(checker, envs, edges, robot, resolution=32):
    checker.upload(envs)
    cfg = checker.launch_config()
    out = {}
    try:
        for persistent in (0, 1):
            checker.set_launch_config(edges_per_cta=64, warps=4, persistent=persistent)
            out[persistent] = checker.check(edges, robot=robot, resolution=resolution)
    finally:
        checker.set_launch_config(**cfg)
    assert np.array_equal(out[0], out[1])
    return out[1]


# 511 .. 513 edges: a probe CTA's batch; 1023 .. 1025, 4097: the offset scan's
# launches and rounds; 255 .. 257 primitives: the ids a voxel
# holds; resolution 1 / 200: one sample block and long edges.
@pytest.mark.parametrize("name,nenv,nedge,resolution", [
    ("uneven", 1, 1, 32), ("uneven", 33, 31, 32), ("uneven", 20, 1023, 32), ("stress", 20, 1024, 32),
    ("stress", 9, 1025, 200), ("uneven", 300, 511, 32), ("stress", 300, 513, 32), ("uneven", 5, 4097, 32), ("plain", 40, 333, 32), ("uneven", 40, 500, 1), ("multi_fetch", 60, 1025, 32),
    ("multi_baxter", 40, 400, 32)])
def test_probed_check_is_the_one_pass_check(checker, name, nenv, nedge, resolution):
    robot = workload.robot_of(name)
    envs = workload.gen_envs(name, nenv, seed=71)
    edges = workload.gen_edges(name, nedge, seed=71)
    got = both(checker, envs, edges, robot, resolution)
    part = slice(0, min(nedge, 60))
    want = orc.check(envs, edges[part], resolution=resolution, robot=robot)
    assert len(orc.adjudicate(envs, edges[part], got[part], want, resolution=resolution, robot=robot)[2]) == 0


@pytest.mark.parametrize("prims", [255, 256, 257, 600])
def test_more_primitives_than_voxel_ids(checker, prims):
    rng = np.random.default_rng(prims)
    c = rng.uniform(-1.0, 1.0, (prims, 3))
    far = {"spheres": make_spheres(c + np.sign(c) * 0.35, rng.uniform(0.02, 0.06, prims))}
    near = {"spheres": make_spheres(c, rng.uniform(0.02, 0.06, prims))}
    both(checker, EnvSet.from_lists([far, near, {}]), workload.gen_edges("uneven", 300, seed=5), "panda")


def test_records_without_a_distance_bound(checker):
    """Axes that stretch distances, a negative radius, non-finite values, and an
    edge that is not a number: the walk decides all of them, as without the probe."""
    rng = np.random.default_rng(3)
    n = 6
    box = make_cuboids(rng.uniform(-0.6, 0.6, (n, 3)), rng.uniform(-3, 3, (n, 3)), rng.uniform(0.02, 0.2, (n, 3)))
    wide, skew, inf = box.copy(), box.copy(), box.copy()
    wide[:, 3:12] *= 2.0
    skew[:, 6:9] = skew[:, 3:6]
    inf[2, 12:15] = np.inf
    neg = make_spheres(rng.uniform(-0.6, 0.6, (n, 3)), np.full(n, -0.3))
    nan = make_spheres(rng.uniform(-0.6, 0.6, (n, 3)), np.full(n, np.nan))
    envs = EnvSet.from_lists([{"cuboids": wide}, {"cuboids": skew}, {"cuboids": inf}, {"spheres": neg},
                              {"spheres": nan}, {"cuboids": box}])
    edges = workload.gen_edges("uneven", 200, seed=6)
    edges[7, :, 3] = np.nan
    both(checker, envs, edges, "panda")


def test_more_pairs_than_the_queue_holds(checker):
    """70 000 environments x 1000 edges: two slabs."""
    n = 70000
    rng = np.random.default_rng(8)
    r = make_spheres(rng.uniform(-0.8, 0.8, (n, 3)) + [0, 0, 0.5], rng.uniform(0.05, 0.15, n))
    envs = EnvSet({"spheres": np.ones(n, np.uint32)}, {"spheres": r})
    both(checker, envs, workload.gen_edges("uneven", 1000, seed=9), "panda")


@pytest.mark.parametrize("prims", [1, 63, 64, 65, 127, 129, 700])
@pytest.mark.parametrize("persistent", [0, 1])
def test_mask_words_hold_every_primitive(checker, prims, persistent):
    """Environments at the edges of the cull's 64-primitive words, between an empty
    one and one of a single primitive: the oracle's verdicts (a primitive missing
    from a mask shows as a collision not found)."""
    rng = np.random.default_rng(prims)
    c = rng.uniform(-0.7, 0.7, (prims, 3)) + [0, 0, 0.4]
    half = prims // 2
    many = {"spheres": make_spheres(c[:half], rng.uniform(0.01, 0.05, half)),
            "cuboids": make_cuboids(c[half:], rng.uniform(-3, 3, (prims - half, 3)),
                                    rng.uniform(0.01, 0.05, (prims - half, 3)))}
    envs = EnvSet.from_lists([{}, many, {"spheres": make_spheres(c[:1], [0.2])}, many])
    edges = workload.gen_edges("uneven", 80, seed=prims)
    cfg = checker.launch_config()
    checker.upload(envs)
    try:
        checker.set_launch_config(persistent=persistent)
        got = checker.check(edges)
    finally:
        checker.set_launch_config(**cfg)
    assert len(orc.adjudicate(envs, edges, got, orc.check(envs, edges))[2]) == 0
    assert np.array_equal(got[:, 1], got[:, 3])


@pytest.mark.parametrize("name,nedge,resolution", [("uneven", 700, 32), ("plain", 150, 32), ("uneven", 200, 1),
                                                   ("plain", 40, 200)])
def test_self_collision_by_segments(checker, name, nedge, resolution):
    """Without primitives a verdict is the edge's self-collision: the oracle's, on
    edges of one block of samples and of many."""
    envs = EnvSet.from_lists([{}])
    edges = workload.gen_edges(name, nedge, seed=77)
    checker.upload(envs)
    got = checker.check(edges, resolution=resolution)
    want = orc.check(envs, edges, resolution=resolution)
    assert 0 < int(got.sum()) < nedge
    assert len(orc.adjudicate(envs, edges, got, want, resolution=resolution)[2]) == 0


@pytest.mark.parametrize("graph", [False, True])
def test_tables_of_an_earlier_call_too_small(graph):
    """A check is queued before its sample total is known to the host, within the
    tables the calls before it left: growing calls, another robot's wider rows, too
    many samples (nothing is written) and a small call after them."""
    import torch
    from bcc.lib import BccError, Checker
    chk = Checker(0)
    envs = workload.gen_envs("uneven", 40, seed=5)
    chk.upload(envs)
    for name, n, resolution in (("uneven", 20, 32), ("uneven", 700, 32), ("plain", 300, 64), ("multi_fetch", 400, 32),
                                ("uneven", 20, 32), ("plain", 600, 200)):
        robot, edges = workload.robot_of(name), workload.gen_edges(name, n, seed=5)
        other = Checker(0)
        other.upload(envs)
        want = other.check(edges, robot=robot, resolution=resolution)
        other.close()
        for _ in range(2):
            assert np.array_equal(chk.check(edges, robot=robot, resolution=resolution, graph=graph), want)
    bad = workload.gen_edges("uneven", 50, seed=6)
    bad[3:8, 1, 2] = np.inf  # 2^20 steps each: beyond the 2^27 samples of a call
    d_edges = torch.from_numpy(bad).cuda()
    out = torch.full((50, 40), 7, dtype=torch.uint8, device="cuda")
    with pytest.raises(BccError):
        chk.check_device(d_edges.data_ptr(), 50, out.data_ptr(), graph=graph)
    torch.cuda.synchronize()
    assert int((out != 7).sum()) == 0
    edges = workload.gen_edges("uneven", 33, seed=7)
    a, b = chk.check(edges, graph=graph), chk.check(edges, graph=graph, order="plain")
    assert np.array_equal(a, b)
    assert len(orc.adjudicate(envs, edges, a, orc.check(envs, edges))[2]) == 0
    chk.close()


def test_grids_are_built_once_a_robot_and_upload(checker):
    """A context that alternates robots builds each one's grids once an upload."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    envs = workload.gen_envs("multi_fetch", 40, seed=91)
    calls = [(r, workload.gen_edges(n, 300, seed=91)) for r, n in (("panda", "uneven"), ("fetch", "multi_fetch"),
                                                                   ("baxter", "multi_baxter"))]
    checker.upload(envs)
    cfg = checker.launch_config()
    checker.set_launch_config(edges_per_cta=64, warps=4, persistent=1)
    try:
        with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
            torch.zeros(1, device="cuda")
            got = [checker.check(edges, robot=robot) for _ in range(3) for robot, edges in calls]
            torch.cuda.synchronize()
    finally:
        checker.set_launch_config(**cfg)
    for k, (robot, edges) in enumerate(calls):
        assert np.array_equal(got[k], got[k + 3]) and np.array_equal(got[k], got[k + 6])
        want = orc.check(envs, edges[:60], robot=robot)
        assert len(orc.adjudicate(envs, edges[:60], got[k][:60], want, robot=robot)[2]) == 0
    names = [e.name for e in prof.events()]
    if not any("walk_kernel" in n for n in names):
        pytest.skip("this profiler does not see the library's kernels")
    assert sum("probe_grid_kernel" in n for n in names) == 3


def _kernels(call):
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        torch.zeros(1, device="cuda")
        call()
        torch.cuda.synchronize()
    names = [e.name for e in prof.events()]
    if not any("fk_staged_kernel" in n for n in names):
        pytest.skip("this profiler does not see the library's kernels")
    return sum("probe_grid_kernel" in n for n in names), sum("walk_kernel" in n for n in names)


@pytest.mark.parametrize("graph", [False, True])
def test_first_check_of_a_small_set_builds_no_grids(graph):
    """A set's grids cost more than they save its first few checks of a middle size:
    those take one pass; a set that goes on being checked is probed, with one build, and
    a new set starts over.  A large first check is probed at once."""
    from bcc.lib import Checker
    chk = Checker(0)
    sets = [workload.gen_envs("uneven", 60, seed=s) for s in (92, 93)]
    edges = workload.gen_edges("uneven", 800, seed=92)
    for envs in sets:
        want = orc.check(envs, edges[:60])
        chk.upload(envs)
        seen = []
        for _ in range(40):
            got = []
            seen.append(_kernels(lambda: got.append(chk.check(edges, graph=graph))))
            if len(seen) in (1, 2, 40):
                assert len(orc.adjudicate(envs, edges[:60], got[0][:60], want)[2]) == 0
        assert seen[0] == (0, 0) and seen[-1] == (0, 1)
        assert sum(g for g, _ in seen) == 1  # then every check is probed
        assert [w for _, w in seen] == sorted(w for _, w in seen)
    chk.close()
    big = Checker(0)
    big.upload(workload.gen_envs("uneven", 600, seed=94))
    edges = workload.gen_edges("uneven", 8000, seed=94)
    assert _kernels(lambda: big.check(edges)) == (1, 1)
    big.close()


def _oracles(envs, edges, got, robot="panda"):
    want = orc.check(envs, edges, robot=robot)
    assert 0 < int(want.sum()) < want.size
    assert len(orc.adjudicate(envs, edges, got, want, robot=robot)[2]) == 0


@pytest.mark.parametrize("prims", [255, 256, 257, 600])
def test_primitives_beyond_voxel_ids_are_the_oracles(checker, prims):
    rng = np.random.default_rng(prims)
    c = rng.uniform(-1.0, 1.0, (prims, 3))
    r = rng.uniform(0.01, 0.03, prims)
    # the nearest primitives are the last ones
    far = {"spheres": make_spheres(np.concatenate([c[:-40] * 0.2 + np.sign(c[:-40]) * 0.9, c[-40:]]), r)}
    envs = EnvSet.from_lists([far, {"spheres": make_spheres(c, r)}, {}])
    edges = workload.gen_edges("uneven", 300, seed=5)
    _oracles(envs, edges, both(checker, envs, edges, "panda"))


def test_pairs_on_both_sides_of_the_queues_slabs_are_the_oracles(checker):
    """70 000 environments x 1000 edges: the first slab ends at environment 67 108."""
    n = 70000
    rng = np.random.default_rng(8)
    r = make_spheres(rng.uniform(-0.8, 0.8, (n, 3)) + [0, 0, 0.5], rng.uniform(0.05, 0.15, n))
    envs = EnvSet({"spheres": np.ones(n, np.uint32)}, {"spheres": r})
    edges = workload.gen_edges("uneven", 1000, seed=9)
    got = both(checker, envs, edges, "panda")
    for lo, hi in ((0, 10), (67098, 67118), (69990, 70000)):
        _oracles(EnvSet({"spheres": np.ones(hi - lo, np.uint32)}, {"spheres": r[lo:hi]}), edges[::5], got[::5, lo:hi])


@pytest.mark.parametrize("name,nenv,nedge", [("uneven", 24, 700), ("stress", 16, 1030), ("multi_fetch", 17, 600),
                                             ("multi_baxter", 11, 520)])
def test_probed_check_is_the_oracles(checker, name, nenv, nedge):
    """Every edge of batches that end within a probe CTA's, not the first ones only
    (three primitives of each kind for the larger robots: with all few edges are free)."""
    robot = workload.robot_of(name)
    envs, edges = workload.gen_envs(name, nenv, seed=73), workload.gen_edges(name, nedge, seed=73)
    if robot != "panda":
        envs = EnvSet.from_lists([{k: r[:3] for k, r in envs.env(i).items()} for i in range(nenv)])
    _oracles(envs, edges, both(checker, envs, edges, robot), robot)
