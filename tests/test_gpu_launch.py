"""GPU tests of the launch machinery: every launch configuration (tile size,
warps, persistent work queue), CUDA-graph replay and the autotuner give the
same verdicts, in both check orders."""
import numpy as np
import pytest

from bcc import mlp, workload

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case(checker):
    envs = workload.gen_envs("uneven", 40, seed=51)
    edges = workload.gen_edges("uneven", 700, seed=51)
    checker.upload(envs)
    checker.mlp_set_params(mlp.init_params(3))
    checker.set_launch_config(edges_per_cta=128, warps=8, persistent=0, queue_min_items=128)
    base = checker.check(edges)
    return envs, edges, base


@pytest.mark.parametrize("lanes", [32, 16])
@pytest.mark.parametrize("tile", [1, 32, 77, 256])
@pytest.mark.parametrize("warps", [4, 8])
@pytest.mark.parametrize("persistent", [0, 1])
def test_launch_configs_agree(checker, case, tile, warps, persistent, lanes):
    """Every launch shape, with a whole warp or a half-warp (16 lanes) per
    walking pair, in both orders (the learned one inline and queued)."""
    envs, edges, base = case
    checker.upload(envs)
    checker.set_launch_config(edges_per_cta=tile, warps=warps, persistent=persistent, queue_min_items=64,
                              lanes=lanes, learned_mode=0, clusters=1)
    for order in ("plain", "learned"):
        assert np.array_equal(checker.check(edges, order=order), base), (tile, warps, persistent, lanes, order)
    checker.set_launch_config(learned_mode=1)
    assert np.array_equal(checker.check(edges, order="learned"), base), (tile, warps, persistent, lanes, "queued")
    checker.set_launch_config(learned_mode=0, lanes=32)


@pytest.mark.parametrize("name,robot", [("uneven", "panda"), ("multi_fetch", "fetch"), ("multi_baxter", "baxter")])
def test_half_warp_walk_keeps_verdicts_and_pairs(checker, name, robot):
    """16 lanes per walking pair: identical verdicts, and the work counters
    count every walked pair and every colliding pair once (robots with
    overhanging leaves keep the whole-warp walk)."""
    envs = workload.gen_envs(name, 30, seed=52)
    edges = workload.gen_edges(name, 400, seed=52)
    checker.upload(envs)
    cfg = checker.launch_config()
    work = {}
    try:
        checker.set_profiling(True, counters=True)
        for lanes in (32, 16):
            checker.set_launch_config(edges_per_cta=64, warps=4, persistent=0, lanes=lanes)
            v = checker.check(edges, robot=robot)
            work[lanes] = (v, checker.work_counters())
    finally:
        checker.set_profiling(False)
        checker.set_launch_config(**cfg)
    assert np.array_equal(work[32][0], work[16][0])
    for k in ("pairs", "candidates", "colliding"):
        assert work[32][1][k] == work[16][1][k], k


def test_graph_replay_agrees(checker, case):
    import torch
    envs, edges, base = case
    checker.upload(envs)
    checker.set_launch_config(edges_per_cta=64, warps=8, persistent=1, queue_min_items=128)
    d_edges = torch.from_numpy(edges).cuda()
    d_res = torch.zeros(base.shape, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    for order in ("plain", "learned"):
        for _ in range(3):  # capture, then replays
            d_res.zero_()
            checker.check_device(d_edges.data_ptr(), len(edges), d_res.data_ptr(), order=order, stream=s, graph=True)
            torch.cuda.synchronize()
            assert np.array_equal(d_res.cpu().numpy(), base), order
    # new edge contents: replayed, or re-captured when the sample total changed
    other = workload.gen_edges("uneven", 700, seed=52)
    d_edges.copy_(torch.from_numpy(other))
    checker.check_device(d_edges.data_ptr(), len(edges), d_res.data_ptr(), stream=s, graph=True)
    torch.cuda.synchronize()
    checker.set_launch_config(persistent=0)
    assert np.array_equal(d_res.cpu().numpy(), checker.check(other))


def test_autotune_picks_a_valid_config(checker, case):
    envs, edges, base = case
    checker.upload(envs)
    cfg = checker.autotune(edges, order="plain")
    assert cfg["edges_per_cta"] in (32, 64, 128, 256) and cfg["warps"] in (4, 8)
    assert np.array_equal(checker.check(edges), base)
    cfg = checker.autotune(edges, order="learned")
    # the learned order's shape, mode, clusters and queue threshold are swept
    assert cfg["edges_per_cta"] in (32, 64, 128, 256) and cfg["warps"] in (4, 8)
    assert cfg["learned_mode"] in (0, 1) and cfg["clusters"] in (1, 4, 8, 16) and cfg["lanes"] in (32, 16)
    if cfg["learned_mode"] == 1:
        assert cfg["queue_min_items"] in (64, 128, 256, 512, 1024, 2048, 4096)
    assert np.array_equal(checker.check(edges, order="learned"), base)


@pytest.mark.parametrize("name,nenv,nedge", [
    ("uneven", 40, 408), ("stress", 1, 64), ("multi_fetch", 40, 400),  # below 2^14 pairs: one pass
    ("uneven", 400, 10000), ("multi_fetch", 500, 5000)])               # records of up to, and above, 8192 bytes: probed
def test_shape_chosen_by_size_survives_a_saved_configuration(name, nenv, nedge):
    """A fresh context's launch shapes: the oracle's verdicts, and the same work (which
    tells the one-pass check from the probed one) after its configuration was saved,
    changed and restored, or set in other values only."""
    from bcc.lib import Checker
    from oracle import oracle as orc
    robot = workload.robot_of(name)
    envs, edges = workload.gen_envs(name, nenv, seed=53), workload.gen_edges(name, nedge, seed=53)
    work = {}
    for how in ("fresh", "restored", "threshold"):
        chk = Checker(0)
        chk.upload(envs)
        chk.set_profiling(True, counters=True)
        cfg = chk.launch_config()
        assert (cfg["edges_per_cta"], cfg["warps"], cfg["persistent"]) == (128, 8, 1)
        if how == "restored":
            for persistent in (0, 1):
                chk.set_launch_config(edges_per_cta=64, warps=4, persistent=persistent)
                work[persistent] = (chk.check(edges, robot=robot), chk.work_counters())
            chk.set_launch_config(**cfg)
        elif how == "threshold":
            chk.set_launch_config(queue_min_items=64)
        got = [chk.check(edges, robot=robot) for _ in range(2)]
        work[how] = (got[1], chk.work_counters())
        assert np.array_equal(got[0], got[1])
        chk.close()
    assert work[0][1]["candidates"] != work[1][1]["candidates"]
    for how in ("fresh", "restored", "threshold"):
        assert work[how][1] == work[1 if nenv * nedge >= 1 << 14 else 0][1], how
        assert np.array_equal(work[how][0], work[1][0])
    part = edges[:80]
    want = orc.check(envs, part, robot=robot)
    assert len(orc.adjudicate(envs, part, work["fresh"][0][:80], want, robot=robot)[2]) == 0


def test_failed_autotune_leaves_the_configuration():
    """No network for the learned order: an error, and the shapes as before it."""
    from bcc.lib import BccError, Checker
    envs, edges = workload.gen_envs("uneven", 30, seed=54), workload.gen_edges("uneven", 300, seed=54)
    chk = Checker(0)
    chk.upload(envs)
    chk.set_profiling(True, counters=True)
    want = chk.check(edges), chk.work_counters()
    with pytest.raises(BccError):
        chk.autotune(edges, order="learned")
    chk.set_profiling(True, counters=True)
    got = chk.check(edges), chk.work_counters()
    assert np.array_equal(got[0], want[0]) and got[1] == want[1]
    chk.close()


def test_first_check_allocates_its_tables_at_once():
    """A first check's device allocations: a fixed few, each a cost of its own; the rows
    and their segments' spheres share one, whatever their sizes."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    from bcc.lib import Checker
    envs, edges = workload.gen_envs("multi_baxter", 4, seed=55), workload.gen_edges("multi_baxter", 3000, seed=55)
    torch.zeros(1, device="cuda")  # the profiled region's own
    chk = Checker(0)
    chk.upload(envs)
    chk.check(edges[:1], robot="baxter")  # the buffers of fixed sizes
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA], acc_events=True) as prof:
        chk.check(edges, robot="baxter")
        torch.cuda.synchronize()
    names = [e.name for e in prof.events()]
    chk.close()
    if not any("cudaLaunchKernel" in x for x in names):
        pytest.skip("this profiler does not see the library's calls")
    assert sum(x == "cudaMalloc" for x in names) == 4  # edges, verdicts, the edges' values, the table


def test_autotune_times_a_probed_shape_once():
    """The probed check has no edge tile: its two warp counts are timed, a check and five
    replays each, not once a tile."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    from bcc.lib import Checker
    envs, edges = workload.gen_envs("uneven", 30, seed=56), workload.gen_edges("uneven", 300, seed=56)
    chk = Checker(0)
    chk.upload(envs)
    want = chk.check(edges)
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        torch.zeros(1, device="cuda")
        chk.autotune(edges, order="plain")
        torch.cuda.synchronize()
    assert np.array_equal(chk.check(edges), want)
    chk.close()
    names = [e.name for e in prof.events()]
    if not any("check_kernel" in n for n in names):
        pytest.skip("this profiler does not see the library's kernels")
    assert sum("probe_kernel" in n for n in names) == 2 * 6


def test_graph_is_captured_once():
    """Equal captured calls of a new context share one graph from the first on; one whose
    edges need a larger table takes another."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    from bcc.lib import Checker
    envs = workload.gen_envs("uneven", 10, seed=57)
    small, large = workload.gen_edges("uneven", 200, seed=57), workload.gen_edges("plain", 200, seed=57)
    chk, other = Checker(0), Checker(0)
    chk.upload(envs)
    other.upload(envs)
    counts = []
    for edges, n in ((small, 3), (large, 3), (small, 2)):
        want = other.check(edges)
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA], acc_events=True) as prof:
            torch.zeros(1, device="cuda")
            for _ in range(n):
                assert np.array_equal(chk.check(edges, graph=True), want)
            torch.cuda.synchronize()
        names = [e.name for e in prof.events()]
        if not any(n.startswith("cudaGraphLaunch") for n in names):
            pytest.skip("this profiler does not see the library's calls")
        counts.append(sum(x.startswith("cudaGraphInstantiate") for x in names))
    chk.close()
    other.close()
    # the larger call queues the graph at hand, finds the table too small, and captures again
    assert counts == [1, 1, 0], counts
