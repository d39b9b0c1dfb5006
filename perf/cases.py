"""The checker's performance cases: the calls its users make, over the sizes
the workload generators, the tests and the benchmark use.

A case is a dict of plain values; `kind` says which public call it makes:

* ``device``   Checker.check_device on device-resident edges and verdicts
               (a planner or sampler that keeps its edges on the GPU);
* ``host``     Checker.check on pinned host arrays (a CPU planner);
* ``oneshot``  Checker.upload of a new environment set followed by
               Checker.check, the shape of the reference's single entry point
               batch_cc::batch_cc (src/batch_cc.hh:4-6), which takes the
               environments with every call;
* ``noalloc``  bcc_check_noalloc on packed records (a real-time thread);
* ``forward``  Checker.mlp_forward_device, scoring of sample configurations;
* ``train``    Checker.mlp_train_step_device, one optimisation step;
* ``grads``    Checker.mlp_gradients_device, gradients back on the host.

Verdicts are bytes; logits, losses, gradients and weights are FP32.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "batch-cc_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

from bcc import lib as bcclib  # noqa: E402
from bcc import mlp, workload  # noqa: E402

CHECKS = ("device", "host", "oneshot", "noalloc")
LR = 2e-3  # the training examples' learning rate
NOALLOC_SAMPLES = 4096  # samples (32 n summed over the edges) bcc_check_noalloc takes per call


def listed():
    return [
        # A control thread validating a handful of local motions in the one
        # environment it currently sees: latency is all that counts.
        dict(name="noalloc_local", kind="noalloc", workload="stress", envs=1, edges=24, resolution=32),
        # A single-query planner checking a batch of candidate motions from the host.
        dict(name="query_host", kind="host", workload="stress", envs=1, edges=64, resolution=32, order="plain",
             graph=False),
        # A mobile manipulator's query over a hundred sensed environments, odd sizes.
        dict(name="fetch_ragged_host", kind="host", workload="multi_fetch", envs=101, edges=1009, resolution=32,
             order="plain", graph=False),
        # The reference's call: environments and edges together, new ones each time.
        dict(name="oneshot_upload", kind="oneshot", workload="uneven", envs=211, edges=997, resolution=32,
             order="plain", graph=False),
        # The plain 100 x 1000 benchmark configuration: long edges (uniform endpoints), replayed graph.
        dict(name="plain_device", kind="device", workload="plain", envs=100, edges=1000, resolution=32,
             order="plain", graph=True),
        # The headline workload, device-resident.
        dict(name="uneven_device", kind="device", workload="uneven", envs=1000, edges=10000, resolution=32,
             order="plain", graph=False),
        # The headline workload end to end from the host in the learned order, network trained on its population.
        dict(name="uneven_learned_host", kind="host", workload="uneven", envs=1000, edges=10000, resolution=32,
             order="learned", graph=True),
        # The multi-robot workloads: many primitives per environment.
        dict(name="fetch_device", kind="device", workload="multi_fetch", envs=500, edges=5000, resolution=32,
             order="plain", graph=False),
        dict(name="baxter_device", kind="device", workload="multi_baxter", envs=500, edges=5000, resolution=32,
             order="plain", graph=False),
        # The stress workload's laws (obstacles in the reachable shell, most pairs free): the largest call.
        dict(name="stress_device", kind="device", workload="stress", envs=2000, edges=50000, resolution=32,
             order="plain", graph=False),
        # Scoring sample configurations in bulk; the row count is no multiple of a tile.
        dict(name="mlp_score", kind="forward", rows=1000003),
        # The training loop's step at its default batch.
        dict(name="mlp_train_step", kind="train", rows=16384),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["device", "device", "device", "host", "host", "oneshot", "noalloc", "forward", "train", "grads"])
    if kind == "forward":
        return dict(kind=kind, rows=_log_int(rng, 1, 4000000))
    if kind in ("train", "grads"):
        return dict(kind=kind, rows=_log_int(rng, 128, 65536))
    if kind == "noalloc":
        return dict(kind=kind, workload=rng.choice(["uneven", "stress"]), envs=_log_int(rng, 8, 64),
                    edges=rng.randint(8, 40), resolution=32)
    name = rng.choice(["plain", "uneven", "uneven", "stress", "multi_fetch", "multi_baxter"])
    small = name == "plain" or kind == "oneshot"
    few = (50, 500) if name.startswith("multi") else (4, 40)  # with that many primitives few motions are free
    return dict(kind=kind, workload=name, envs=_log_int(rng, few[0], 300 if small else 1000),
                edges=_log_int(rng, few[1], 3000 if small else 10000), resolution=rng.choice([32, 32, 32, 16, 64]),
                order="learned" if kind != "oneshot" and rng.random() < 0.25 else "plain",
                graph=kind != "oneshot" and rng.random() < 0.5)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _mlp_rows(rows, seed):
    """Feature rows as the checker builds them (joints in [-1, 1], environment
    code, position along the edge, bias input 0), BF16 bits, and labels."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.zeros(rows, mlp.IN, device="cuda")
    x[:, :7] = torch.rand(rows, 7, device="cuda", generator=g) * 2 - 1
    x[:, 7:11] = torch.rand(rows, 4, device="cuda", generator=g)
    x[:, 11:35] = torch.rand(rows, 24, device="cuda", generator=g) * 2 - 0.5
    x[:, 35:39] = torch.rand(rows, 4, device="cuda", generator=g) * 0.6
    x[:, 46] = torch.rand(rows, device="cuda", generator=g) * 2 - 1
    y = (x[:, 0] + 0.5 * x[:, 3] - x[:, 12] + 0.5 * x[:, 46]
         + 0.5 * torch.randn(rows, device="cuda", generator=g) > 0).to(torch.uint8)
    return x.to(torch.bfloat16), y


def _params(seed):
    p = mlp.init_params(seed % 1000003)
    rng = np.random.default_rng(seed)
    q = mlp.unflatten(p)
    for k in ("b1", "b2", "b3", "b4"):
        q[k][:] = rng.normal(0, 0.05, q[k].shape)
    return p


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _pack(envs):
    L = bcclib.lib()
    soa = envs.as_ctypes()
    n, most = ctypes.c_int64(0), ctypes.c_int32(0)
    L.bcc_pack_envs(ctypes.byref(soa), None, None, ctypes.byref(n), ctypes.byref(most))
    rec = np.zeros((max(n.value, 1), 20), np.float32)
    off = np.zeros(envs.num_envs + 1, np.int32)
    L.bcc_pack_envs(ctypes.byref(soa), rec.ctypes.data_as(ctypes.POINTER(ctypes.c_float)),
                    off.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), ctypes.byref(n), ctypes.byref(most))
    return torch.from_numpy(rec).cuda(), torch.from_numpy(off).cuda(), most.value


def _noalloc():
    f = bcclib.lib().bcc_check_noalloc
    vp = ctypes.c_void_p
    f.argtypes = [ctypes.c_int, vp, vp, ctypes.c_int32, ctypes.c_int32, vp, ctypes.c_int32, ctypes.c_int32, vp, vp]
    f.restype = ctypes.c_int
    return f


def prepare(case, seed):
    kind = case["kind"]
    if kind not in CHECKS:
        x, y = _mlp_rows(case["rows"], seed)
        p = _params(seed)
        chk = bcclib.Checker(0)
        chk.mlp_set_params(p)
        return dict(case=case, chk=chk, x=x, y=y, logits=torch.empty(case["rows"], device="cuda"))
    name, N, E = case["workload"], case["envs"], case["edges"]
    envs = workload.gen_envs(name, N, seed=seed)
    edges = workload.gen_edges(name, E, seed=seed)
    s = dict(case=case, robot=workload.robot_of(name))
    if kind == "noalloc":
        s["rec"], s["off"], s["most"] = _pack(envs)
        keep, rows = [], 0  # as many of the edges as the entry point's sample limit takes
        for e in edges:
            rows += bcclib.edge_samples(e[0], e[1], case["resolution"])
            if rows > NOALLOC_SAMPLES:
                break
            keep.append(e)
        s["edges"] = torch.from_numpy(np.stack(keep)).cuda()
        s["out"] = torch.empty((len(keep), N), dtype=torch.uint8, device="cuda")
        s["call"] = _noalloc()
        return s
    chk = s["chk"] = bcclib.Checker(0)
    if case["order"] == "learned":
        chk.mlp_set_params(mlp.init_params(seed % 1000003))
        if name in ("uneven", "stress") and N * E >= 1000000:
            # a network trained on this workload's own population, other environments and edges
            chk.upload(workload.gen_envs(name, 200, seed=seed + 1000000007))
            chk.mlp_train_queued(workload.gen_edges(name, 1000, seed=seed + 1000000007), num_samples=1 << 17,
                                 queue_min_items=128, epochs=1, batch=2048, lr=LR, seed=seed % 1000003,
                                 robot=s["robot"])
    if kind == "oneshot":
        s["envs"] = envs
    else:
        chk.upload(envs)
    if kind == "device":
        s["edges"] = torch.from_numpy(edges).cuda()
        s["out"] = torch.empty((E, N), dtype=torch.uint8, device="cuda")
    else:
        pe = _pinned(edges.shape, torch.float32)
        pe.copy_(torch.from_numpy(edges))
        s["keep"] = (pe, _pinned((E, N), torch.uint8))
        s["edges"], s["out"] = s["keep"][0].numpy(), s["keep"][1].numpy()
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forward":
        state["chk"].mlp_forward_device(state["x"].data_ptr(), case["rows"], state["logits"].data_ptr(),
                                        stream=_stream())
        return state["logits"]
    if kind == "train":
        loss = state["chk"].mlp_train_step_device(state["x"].data_ptr(), state["y"].data_ptr(), case["rows"], LR)
        return dict(loss=loss, params=state["chk"].mlp_get_params())
    if kind == "grads":
        g, loss = state["chk"].mlp_gradients_device(state["x"].data_ptr(), state["y"].data_ptr(), case["rows"])
        return dict(loss=loss, grads=g)
    if kind == "noalloc":
        st = state["call"](bcclib.ROBOTS[state["robot"]], state["rec"].data_ptr(), state["off"].data_ptr(),
                           case["envs"], state["most"], state["edges"].data_ptr(), len(state["edges"]),
                           case["resolution"], state["out"].data_ptr(), ctypes.c_void_p(_stream()))
        if st:
            raise bcclib.BccError(st, "bcc_check_noalloc")
        return state["out"]
    chk = state["chk"]
    if kind == "device":
        chk.check_device(state["edges"].data_ptr(), case["edges"], state["out"].data_ptr(),
                         resolution=case["resolution"], robot=state["robot"], order=case["order"], stream=_stream(),
                         graph=case["graph"])
        return state["out"]
    if kind == "oneshot":
        chk.upload(state["envs"])
    return chk.check(state["edges"], resolution=case["resolution"], robot=state["robot"], order=case["order"],
                     out=state["out"], graph=case["graph"])


def work(case):
    if case["kind"] not in CHECKS:
        rows = case["rows"]
        mac = mlp.IN * mlp.HID + 2 * mlp.HID * mlp.HID + mlp.HID
        if case["kind"] == "forward":
            return {"bytes": rows * (mlp.IN * 2 + 4) + 4 * mlp.NUM_PARAMS, "flops": 2.0 * rows * mac}
        # forward, weight gradients, and the gradients of the two hidden inputs
        back = mac + 2 * mlp.HID * mlp.HID + mlp.HID
        state = 6 if case["kind"] == "train" else 2  # weights and moments in and out, or weights in, gradients out
        return {"bytes": rows * (mlp.IN * 2 + 1) + 4 * state * mlp.NUM_PARAMS, "flops": 2.0 * rows * (mac + back)}
    w = workload.WORKLOADS[case["workload"]]
    prims = 20 if w["prims"] == "fixed" else sum(w["prims"]) / 2
    dof = workload.DOF[w["robot"]]
    # edges and primitive records (40 % spheres of 4 floats, 40 % cuboids of 15, 20 % capsules of 8) in, verdicts out
    return {"bytes": case["edges"] * 2 * dof * 4 + case["envs"] * prims * 4 * (0.4 * 4 + 0.4 * 15 + 0.2 * 8)
            + case["envs"] * case["edges"], "flops": 0}


def _forward64(P, x):
    h = []
    z = x
    for k in (1, 2, 3):
        z = torch.relu(z @ P["W%d" % k] + P["b%d" % k])
        h.append(z)
    return z @ P["w4"] + P["b4"], h


def exact(case, seed):
    if case["kind"] in CHECKS:
        return None  # verdicts are bytes
    x, y = _mlp_rows(case["rows"], seed)
    p = _params(seed)
    P = {k: torch.from_numpy(v.astype(np.float64)).cuda() for k, v in mlp.unflatten(p).items()}
    grads = {k: torch.zeros_like(v) for k, v in P.items()}
    rows, loss, logits = case["rows"], 0.0, []
    for a in range(0, rows, 1 << 18):
        xx, yy = x[a:a + (1 << 18)].double(), y[a:a + (1 << 18)].double()
        z, h = _forward64(P, xx)
        if case["kind"] == "forward":
            logits.append(z)
            continue
        loss += float((torch.clamp(z, min=0) - z * yy + torch.log1p(torch.exp(-z.abs()))).sum())
        d = (torch.sigmoid(z) - yy) / rows
        grads["b4"] += d.sum()
        grads["w4"] += h[2].T @ d
        d = d[:, None] * P["w4"] * (h[2] > 0)
        for k in (3, 2, 1):
            grads["b%d" % k] += d.sum(0)
            grads["W%d" % k] += (h[k - 2] if k > 1 else xx).T @ d
            if k > 1:
                d = (d @ P["W%d" % k].T) * (h[k - 2] > 0)
    if case["kind"] == "forward":
        return torch.cat(logits)
    flat = torch.cat([grads[k].reshape(-1) for k, _ in mlp.SHAPES]).cpu().numpy()
    if case["kind"] == "grads":
        return dict(loss=loss, grads=flat)
    # Adam's first step: both moments' bias corrections cancel their decay
    return dict(loss=loss, params=p.astype(np.float64) - LR * flat / (np.abs(flat) + 1e-8))
