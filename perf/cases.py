"""Performance cases of the Gravity-Sim force-and-integrate path.

Each case is one pass of a user's program through the public entry points: upload a
system from pinned host arrays (gs_set_particles), advance it (gs_run), read it back
(gs_get_particles); or one step on device buffers the caller owns
(gs_direct_step_noalloc); or a batch of independent systems (gs_batch_run); or a request
trace through the serving loop (gs_server_run_trace).  Sizes, generators and parameters
are those of the repository's benchmark and tests.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "gravity-sim_gb300")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)
import gsim  # noqa: E402

DT, SOFTENING, SIZE = 1e-3, 0.2, 100.0
GENERATORS = {"random": gsim.GEN_RANDOM, "galaxy": gsim.GEN_GALAXY, "collision": gsim.GEN_GALAXY_COLLISION,
              "disk": gsim.GEN_UNIFORM_DISK, "spiral": gsim.GEN_SPIRAL, "two_disks": gsim.GEN_EXP_DISK_COLLISION}
RELATIVE = gsim.FLAGS_ACCURATE | gsim.FLAG_RELATIVE_MAC
CROSSOVER = 2048  # direct sum below, Barnes-Hut from here on, in batches and in the serving loop
EXACT_PAIRS = 6e10  # pair evaluations a 64-bit direct sum makes in well under 20 seconds


def _modes():
    """The ways a system is run: the library's parameters of each."""
    return {
        "direct": dict(algorithm=gsim.DIRECT_SUM),  # FP32 tiles, compensated sums
        "direct_reference": dict(algorithm=gsim.DIRECT_SUM, math_mode=gsim.MATH_REFERENCE),  # the shader's order
        "rule": dict(algorithm=gsim.BARNES_HUT),  # the drop-in defaults: fixed box, monopoles, theta = 1
        "theta": dict(algorithm=gsim.BARNES_HUT, box_mode=gsim.BOX_BOUNDING, accuracy_parameter=0.35,
                      flags=gsim.FLAGS_ACCURATE),  # accurate mode, geometric criterion
        "relative": dict(algorithm=gsim.BARNES_HUT, box_mode=gsim.BOX_BOUNDING, accuracy_parameter=1.0,
                         relative_accuracy=0.006, relative_theta_floor=0.2, flags=RELATIVE),  # <= 1e-3 force error
    }


def listed():
    return [
        # a host application's own buffers, one small step: launch and latency
        dict(name="noalloc_1k", path="noalloc", n=1024, kind="disk"),
        # a small interactive scene at an odd size, many steps between readbacks
        dict(name="direct_1000", path="single", mode="direct", n=1000, kind="random", steps=100, key_bits=12),
        # the reference's own small configuration: 4096 particles on a disk at rest, 10 steps
        dict(name="direct_4096", path="single", mode="direct", n=4096, kind="disk", steps=10, key_bits=12),
        # the precision study's two-disk collision, where the O(N^2) arithmetic is everything
        dict(name="direct_50k", path="single", mode="direct", n=50000, kind="two_disks", steps=4, key_bits=12),
        # parity runs: the shader's summation order with correctly rounded 1/sqrt
        dict(name="direct_reference_4096", path="single", mode="direct_reference", n=4096, kind="disk", steps=10,
             key_bits=12),
        # Barnes-Hut with the drop-in defaults on a small galaxy: launches of the step's many stages
        dict(name="rule_3k", path="single", mode="rule", n=3000, kind="galaxy", steps=50, key_bits=12),
        # the same defaults at the benchmark's full size
        dict(name="rule_500k", path="single", mode="rule", n=500000, kind="spiral", steps=10, key_bits=12),
        # the accurate criterion on a mid-size system (the common size of batched and served members)
        dict(name="relative_20k", path="single", mode="relative", n=20000, kind="disk", steps=20, key_bits=12),
        # accurate mode by opening angle alone
        dict(name="theta_100k", path="single", mode="theta", n=100000, kind="spiral", steps=5, key_bits=12),
        # the headline: 500k spiral, relative criterion
        dict(name="relative_500k", path="single", mode="relative", n=500000, kind="spiral", steps=10, key_bits=12),
        # many independent systems of uneven size in one launch per stage
        dict(name="batch_64", path="batch", count=64, lo=1024, hi=262144, steps=5),
        # requests that arrive together, run through continuous batching
        dict(name="served_12", path="served", count=12, lo=2048, hi=131072, steps_lo=10, steps_hi=50),
    ]


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    path = rng.choice(["noalloc", "single", "single", "single", "single", "single", "batch", "served"])
    if path == "noalloc":
        return dict(path=path, n=64 * _log_uniform(rng, 1, 1024), kind=rng.choice(["disk", "spiral", "random"]))
    if path == "batch":
        return dict(path=path, count=rng.randint(8, 56), lo=1024, hi=_log_uniform(rng, 8192, 131072),
                    steps=rng.randint(2, 5))
    if path == "served":
        return dict(path=path, count=rng.randint(4, 10), lo=2048, hi=_log_uniform(rng, 16384, 65536), steps_lo=5,
                    steps_hi=rng.randint(10, 30))
    mode = rng.choice(["direct", "direct", "direct_reference", "rule", "rule", "theta", "relative", "relative"])
    if mode.startswith("direct"):
        n = _log_uniform(rng, 64, 50000 if mode == "direct" else 8192)
        return dict(path=path, mode=mode, n=n, kind=rng.choice(["random", "disk", "two_disks"]),
                    steps=100 if n < 2048 else 10 if n < 16384 else 3, key_bits=12)
    n = _log_uniform(rng, 1000, 450000)
    return dict(path=path, mode=mode, n=n, kind=rng.choice(["galaxy", "spiral", "collision"]),
                steps=20 if n < 32768 else 5, key_bits=rng.choice([12, 12, 12, 15]))


def _params(mode, key_bits=12):
    kw = dict(_modes()[mode])
    if kw.get("box_mode") == gsim.BOX_BOUNDING:
        kw["key_bits"] = key_bits
    return gsim.default_params(simulation_time=DT, softening_len=SOFTENING, **kw)


def _make(kind, n, seed):
    return gsim.generate(GENERATORS[kind], n, size=SIZE, seed=seed)


def _members(case, seed):
    """(generator, N, seed) of each member of a batch, or each request of a trace."""
    rng = np.random.default_rng(1004)
    n = np.floor(np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), case["count"]))).astype(int)
    kinds = ["disk", "spiral"] if case["path"] == "batch" else ["disk", "spiral", "two_disks"]
    return [(kinds[int(k)], int(m), 1000 * seed + j)
            for j, (k, m) in enumerate(zip(rng.integers(0, len(kinds), case["count"]), n))]


def _steps(case):
    """Steps of each request of a trace."""
    return [int(x) for x in np.random.default_rng(1005).integers(case["steps_lo"], case["steps_hi"] + 1,
                                                                 case["count"])]


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float32, pin_memory=True)
    t.copy_(torch.from_numpy(a))
    return t


def _pointer(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_float))


def _check(status):
    if status:
        raise gsim.GsimError(status, gsim.lib().gs_last_error().decode())


def _noalloc():
    f = gsim.lib().gs_direct_step_noalloc
    f.argtypes = [C.c_void_p] * 5 + [C.c_uint64, C.c_float, C.c_float, C.c_float, C.c_void_p]
    f.restype = C.c_int
    return f


def prepare(case, seed):
    if case["path"] == "noalloc":
        pos, vel, mass = _make(case["kind"], case["n"], seed)
        dev = [torch.from_numpy(a).cuda() for a in (pos, vel, mass)]
        return dict(path="noalloc", n=case["n"], step=_noalloc(), inputs=dev,
                    outputs=[torch.empty_like(dev[0]), torch.empty_like(dev[1])])
    if case["path"] == "single":
        arrays = [_pinned(a) for a in _make(case["kind"], case["n"], seed)]
        sim = gsim.Simulation(*[a.numpy() for a in arrays], params=_params(case["mode"], case["key_bits"]))
        return dict(path="single", sim=sim, steps=case["steps"], inputs=arrays, views=[a.numpy() for a in arrays],
                    outputs=[torch.empty_like(a).pin_memory() for a in arrays])
    if case["path"] == "batch":
        made = [_make(*m) for m in _members(case, seed)]
        total = sum(len(m[2]) for m in made)
        inputs = [torch.empty((total, 2), pin_memory=True), torch.empty((total, 2), pin_memory=True),
                  torch.empty(total, pin_memory=True)]
        outputs = [torch.empty_like(t).pin_memory() for t in inputs]
        sims, views, slots, at = [], [], [], 0
        for arrays in made:
            n = len(arrays[2])
            for t, a in zip(inputs, arrays):
                t[at:at + n].copy_(torch.from_numpy(a))
            views.append([t[at:at + n].numpy() for t in inputs])
            slots.append([t[at:at + n] for t in outputs])
            sims.append(gsim.Simulation(*views[-1], params=_params("direct" if n < CROSSOVER else "relative")))
            at += n
        return dict(path="batch", sims=sims, batch=gsim.Batch(sims), steps=case["steps"], inputs=inputs, views=views,
                    slots=slots, outputs=outputs)
    made = [[np.ascontiguousarray(a) for a in _make(*m)] for m in _members(case, seed)]
    requests = []
    for (pos, vel, mass), steps in zip(made, _steps(case)):
        r = gsim.make_request(len(mass), steps)
        r.pos_xy, r.vel_xy, r.mass = (a.ctypes.data_as(C.POINTER(C.c_float)) for a in (pos, vel, mass))
        requests.append(r)
    server = gsim.Server(64 << 30, CROSSOVER, _params("direct"), _params("relative"), keep_results=True)
    return dict(path="served", server=server, requests=requests, arrivals=[0.0] * len(requests), inputs=made)


def run(state):
    if state["path"] == "noalloc":
        (pos, vel, mass), (pos_out, vel_out) = state["inputs"], state["outputs"]
        _check(state["step"](pos.data_ptr(), vel.data_ptr(), mass.data_ptr(), pos_out.data_ptr(), vel_out.data_ptr(),
                             state["n"], 1.0, DT, SOFTENING, torch.cuda.current_stream().cuda_stream))
        return state["outputs"]
    if state["path"] == "single":
        sim = state["sim"]
        sim.set_particles(*state["views"])
        sim.run(state["steps"])
        _check(gsim.lib().gs_get_particles(sim.handle, *[_pointer(t) for t in state["outputs"]]))
        return state["outputs"]
    if state["path"] == "batch":
        for sim, view in zip(state["sims"], state["views"]):
            sim.set_particles(*view)
        state["batch"].run(state["steps"])
        for sim, slot in zip(state["sims"], state["slots"]):
            _check(gsim.lib().gs_get_particles(sim.handle, *[_pointer(t) for t in slot]))
        return state["outputs"]
    ids = state["server"].run_trace(state["requests"], state["arrivals"], timeout_s=60.0)
    return [list(state["server"].result(i)) for i in ids]


# Interactions a particle sums per step, times the operations of one (14 for a monopole, 33
# with the quadrupole term), per doubling of N: 184 monopoles at N = 500k under the
# reference's rule, 554 (half of them nodes) by the relative criterion, 670 at theta = 0.35.
PER_DOUBLING = {"rule": 9.7 * 14, "relative": 29.3 * 23, "theta": 35.4 * 23}


def _flops(mode, n, steps):
    if mode.startswith("direct"):
        return 14.0 * n * n * steps
    return PER_DOUBLING[mode] * math.log2(max(n, 2)) * n * steps


def work(case):
    """Each state array read once and written once, and the arithmetic of the interactions."""
    if case["path"] == "noalloc":
        return {"bytes": 36.0 * case["n"], "flops": _flops("direct", case["n"], 1)}
    if case["path"] == "single":
        return {"bytes": 40.0 * case["n"], "flops": _flops(case["mode"], case["n"], case["steps"])}
    sizes = [m[1] for m in _members(case, 0)]
    steps = [case["steps"]] * len(sizes) if case["path"] == "batch" else _steps(case)
    return {"bytes": 40.0 * sum(sizes),
            "flops": sum(_flops("direct" if n < CROSSOVER else "relative", n, k) for n, k in zip(sizes, steps))}


def _advance64(pos, vel, mass, steps):
    """The same steps by the direct sum in 64 bits."""
    p, v, m = (torch.from_numpy(a).cuda().double() for a in (pos, vel, mass))
    eps2 = float(np.float32(SOFTENING) * np.float32(SOFTENING))
    dt = float(np.float32(DT))
    rows = max(1, int(2 ** 26 // len(m)))
    for _ in range(steps):
        x, y = p[:, 0].contiguous(), p[:, 1].contiguous()
        acc = torch.empty_like(p)
        for i in range(0, len(m), rows):
            dx, dy = x[None, :] - x[i:i + rows, None], y[None, :] - y[i:i + rows, None]
            s = dx * dx
            s.addcmul_(dy, dy).add_(eps2).pow_(-1.5).mul_(m)
            acc[i:i + rows, 0] = (dx.mul_(s)).sum(1)
            acc[i:i + rows, 1] = (dy.mul_(s)).sum(1)
        v1 = v + acc * dt
        p = p + (v + v1) * (0.5 * dt)
        v = v1
    return [p, v, m]


def exact(case, seed):
    if case["path"] == "batch":
        members, steps = _members(case, seed), [case["steps"]] * case["count"]
    elif case["path"] == "served":
        members, steps = _members(case, seed), _steps(case)
    else:
        members, steps = [(case["kind"], case["n"], seed)], [case.get("steps", 1)]
    if sum(float(n) * n * k for (_, n, _), k in zip(members, steps)) > EXACT_PAIRS:
        return None
    made = [_advance64(*_make(*m), k) for m, k in zip(members, steps)]
    if case["path"] == "noalloc":
        return made[0][:2]
    if case["path"] == "single":
        return made[0]
    if case["path"] == "batch":
        return [torch.cat([m[j] for m in made]) for j in range(3)]
    return made
