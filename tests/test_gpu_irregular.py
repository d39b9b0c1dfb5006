"""GPU tests of environments whose records are not boxes: axes that stretch, shrink
or skew, negative radii, values that are not finite.  No bound on distances holds
there, so every entry point and check order is compared with the oracle, which
makes the reference's tests as they stand."""
import ctypes

import numpy as np
import pytest

from bcc import EnvSet, mlp, workload
from bcc import lib as bcclib
from bcc.workload import make_capsules, make_cuboids, make_spheres
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
ROBOT = {"panda": "uneven", "fetch": "multi_fetch", "baxter": "multi_baxter"}


def _cuboids(rng, n, reach):
    return make_cuboids(rng.uniform(-reach, reach, (n, 3)) + [0, 0, 0.5 * reach], rng.uniform(-3, 3, (n, 3)),
                        rng.uniform(0.02, 0.2, (n, 3)))


def _axes(box, f):
    box[:, 3:12] = f(box[:, 3:12].reshape(-1, 3, 3).astype(np.float64)).reshape(-1, 9)
    return box


def _kind(name, rng, reach):
    n = 8
    box = _cuboids(rng, n, reach)
    c = rng.uniform(-reach, reach, (n, 3)) + [0, 0, 0.5 * reach]
    if name == "wide2":
        return {"cuboids": _axes(box, lambda a: 2.0 * a)}
    if name == "wide3":
        return {"cuboids": _axes(box, lambda a: 3.0 * a)}
    if name == "one_axis":
        return {"cuboids": _axes(box, lambda a: a * np.array([[1.0], [2.5], [1.0]]))}
    if name == "narrow":
        return {"cuboids": _axes(box, lambda a: 0.6 * a)}
    if name == "skew":
        return {"cuboids": _axes(box, lambda a: a + 0.5 * a[:, [1, 2, 0]])}
    if name == "parallel":  # two equal axes: a box without an end in one direction
        box[:, 6:9] = box[:, 3:6]
        return {"cuboids": box[:2], "spheres": make_spheres(c[:2], [0.1, 0.1])}
    if name == "tilted_z":  # a tilted box among the z-aligned ones: its axes are projected
        return {"z_cuboids": box}
    if name == "negative":
        return {"spheres": make_spheres(c, np.full(n, -0.25)),
                "capsules": make_capsules(c, rng.uniform(-3, 3, (n, 3)), np.full(n, -0.2), rng.uniform(0.1, 0.4, n))}
    if name == "not_finite":
        box[0, 12] = np.inf
        sph = make_spheres(c, rng.uniform(0.05, 0.1, n))
        sph[0, 0], sph[1, 3], sph[2, 2] = np.nan, np.nan, np.inf
        cap = make_capsules(c, rng.uniform(-3, 3, (n, 3)), rng.uniform(0.03, 0.08, n), rng.uniform(0.1, 0.4, n))
        cap[0, 4], cap[1, 1], cap[2, 6] = np.nan, np.inf, np.nan
        return {"cuboids": box[:2], "spheres": sph, "capsules": cap}
    return {"cuboids": box}  # "box": regular


KINDS = ("wide2", "wide3", "one_axis", "narrow", "skew", "parallel", "tilted_z", "negative", "not_finite", "box")


def _case(robot, edges=120):
    rng = np.random.default_rng(17)
    reach = 0.7 if robot == "panda" else 1.0
    envs = EnvSet.from_lists([_kind(k, rng, reach) for k in KINDS for _ in range(3)] + [{}])
    return envs, workload.gen_edges(ROBOT[robot], edges, seed=6)


def _is_the_oracles(envs, edges, got, robot, want):
    for i, k in enumerate(KINDS):
        env = slice(3 * i, 3 * i + 3)
        sub = envs.subset(range(env.start, env.stop))
        _, _, bad = orc.adjudicate(sub, edges, got[:, env], want[:, env], robot=robot)
        assert len(bad) == 0, (k, len(bad), int((got[:, env] < want[:, env]).sum()))
    assert np.array_equal(got[:, -1], want[:, -1])


@pytest.mark.parametrize("robot", ["panda", "fetch", "baxter"])
def test_every_check_of_irregular_environments_is_the_oracles(robot):
    envs, edges = _case(robot)
    want = orc.check(envs, edges, robot=robot)
    both = [k for i, k in enumerate(KINDS) if 0 < want[:, 3 * i:3 * i + 3].mean() < 1]
    assert {"wide2", "wide3", "one_axis", "negative", "box"} <= set(both), both
    chk = bcclib.Checker(0)
    chk.upload(envs)
    chk.mlp_set_params(mlp.init_params(5))
    chk.set_profiling(True, counters=True)
    free = int(edges.shape[0] * envs.num_envs)
    for shape in (None, dict(edges_per_cta=32, warps=8, persistent=0), dict(edges_per_cta=64, warps=4, persistent=1)):
        if shape:
            chk.set_launch_config(**shape)
        got = chk.check(edges, robot=robot)
        _is_the_oracles(envs, edges, got, robot, want)
        w = chk.work_counters()
        assert w["pairs"] <= free and w["colliding"] <= w["pairs"]
    chk.set_profiling(False)
    for mode, graph in ((0, False), (0, True), (1, False), (1, True)):
        chk.set_launch_config(learned_mode=mode, queue_min_items=0)
        assert np.array_equal(chk.check(edges, robot=robot, order="learned", graph=graph), got), (mode, graph)
    # a regular set after an irregular one
    plain = workload.gen_envs(ROBOT[robot], 4, seed=3)
    chk.upload(plain)
    got = chk.check(edges, robot=robot)
    assert len(orc.adjudicate(plain, edges, got, orc.check(plain, edges, robot=robot), robot=robot)[2]) == 0
    chk.close()


@pytest.mark.parametrize("robot", ["panda", "fetch", "baxter"])
def test_packed_irregular_records_are_the_oracles(robot):
    import torch
    envs, edges = _case(robot, 100)
    rows = np.cumsum([32 * orc.edge_n(e[0], e[1]) for e in edges])
    edges = edges[:int((rows <= 4096).sum())]
    L = bcclib.lib()
    soa = envs.as_ctypes()
    n, most = ctypes.c_int64(0), ctypes.c_int32(0)
    fp, ip = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_int32)
    assert L.bcc_pack_envs(ctypes.byref(soa), None, None, ctypes.byref(n), ctypes.byref(most)) == 0
    rec, off = np.zeros((n.value, 20), np.float32), np.zeros(envs.num_envs + 1, np.int32)
    assert L.bcc_pack_envs(ctypes.byref(soa), rec.ctypes.data_as(fp), off.ctypes.data_as(ip), ctypes.byref(n),
                           ctypes.byref(most)) == 0
    vp = ctypes.c_void_p
    f = L.bcc_check_noalloc
    f.argtypes = [ctypes.c_int, vp, vp, ctypes.c_int32, ctypes.c_int32, vp, ctypes.c_int32, ctypes.c_int32, vp, vp]
    d_rec, d_off, d_edges = (torch.from_numpy(a).cuda() for a in (rec, off, edges))
    out = torch.full((len(edges), envs.num_envs), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert f(bcclib.ROBOTS[robot], d_rec.data_ptr(), d_off.data_ptr(), envs.num_envs, most.value, d_edges.data_ptr(),
             len(edges), 32, out.data_ptr(), None) == 0
    _is_the_oracles(envs, edges, out.cpu().numpy(), robot, orc.check(envs, edges, robot=robot))


def test_edges_that_are_not_numbers_hit_nothing(checker):
    """As in environments of boxes: a link whose place is not a number is nowhere."""
    envs, edges = _case("panda", 40)
    edges[::2, 1, 0] = np.nan  # the first joint: every link
    checker.upload(envs)
    got = checker.check(edges)
    assert not got[::2].any() and got[1::2].any()
