"""Workloads of the engine's main path through its public Python binding (gcs.py).

listed() names the fixed cases, draw() gives more of the same ranges, prepare()
makes a case's inputs and context from a seed, run() makes one pass, work()
states what a pass cannot do without and exact() gives the outputs in 64 bits
where that is affordable.

Every initial condition is the seeded two-galaxy recipe of the package's own
generator.  The device cases share one CUDA stream, as a program with several
contexts on one GPU would; a step advances its context's state, and the host
cases read the same host Stars on every pass.
"""
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "galaxy-collision-simulator_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import gcs  # noqa: E402
import workloads  # noqa: E402

# The largest listed case bounds what draw() may ask for.
MAX_COST = 1.3e11
# FP64 pair sums of exact() beyond this many pairs take too long.
MAX_PAIRS = 3.0e11


def listed():
    return [
        # A quick look at a small pair: one eager step of a tiny context, where
        # launches and latency are everything.
        dict(name="step_1k", kind="step", n=1408, theta=0.5, eps=0.05, dt=0.005, leaf=8, batch=0, width=32,
             com_fp64=1, graphs=0),
        # The small run of the recipe: 45,056 particles, 200 graph-captured steps.
        dict(name="step_45k", kind="step", n=45056, theta=0.5, eps=0.05, dt=0.005, leaf=8, batch=64, width=32,
             com_fp64=1, graphs=1),
        # The headline: 1,048,576 particles at theta 0.5, graph-captured steps.
        dict(name="step_1m", kind="step", n=1048576, theta=0.5, eps=0.02, dt=0.0025, leaf=4, batch=64, width=32,
             com_fp64=1, graphs=1),
        # The same run at theta 0.7, at an odd size, eager steps, FP32 centres of mass.
        dict(name="step_777k_t07", kind="step", n=777777, theta=0.7, eps=0.02, dt=0.0025, leaf=8, batch=32, width=32,
             com_fp64=0, graphs=0),
        # The precision study: 4,194,304 particles, accelerations with potentials.
        dict(name="accels_4m_pot", kind="accels", n=4194304, theta=0.5, eps=0.01, leaf=8, batch=64, width=32,
             com_fp64=1),
        # Independent collisions of uneven sizes advanced together, 64-target groups.
        dict(name="batched_32", kind="batched", count=32, n_lo=4096, n_hi=262144, mix=0, theta=0.5, eps=0.02,
             dt=0.0025, leaf=8, batch=64, width=64, com_fp64=1),
        # Live mode with the reference's own settings (theta 1, eps^2 10, one
        # particle a leaf, caller bounds, colour map): 300,000 particles, each
        # step's Stars copied to pageable host memory.
        dict(name="live_300k", kind="live", n=300000),
        # Host Stars to host Stars in pinned memory, 1,048,576 particles.
        dict(name="host_1m", kind="host", n=1048576, theta=0.5, eps=0.02, dt=0.0025, leaf=4, batch=64, pinned=1),
        # A burst of small requests through the continuous-batching server.
        dict(name="served_8", kind="served", count=8, n_lo=8192, n_hi=65536, mix=1, steps_lo=3, steps_hi=6,
             slots=4, theta=0.5, eps=0.02, dt=0.0025, leaf=8, batch=64),
        # The allocation-free pair sort at its largest size.
        dict(name="sort_1m", kind="sort", n=1048576),
        # One 1920 x 1080 frame of 1,048,576 particles, read back to the host.
        dict(name="render_1m", kind="render", n=1048576, w=1920, h=1080),
        # The FP64 direct sum that states the force error: a subset of targets.
        dict(name="direct_4k_of_262k", kind="direct", n=262144, targets=4096, eps=0.02),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        case = _draw_one(rng)
        if _cost(case) <= MAX_COST:
            return case


def _draw_one(rng):
    kind = rng.choice(["step", "step", "step", "step", "accels", "batched", "live", "host", "served", "sort",
                       "render", "direct"])
    theta = rng.choice([0.5, 0.7])
    eps = rng.choice([0.01, 0.02, 0.05])
    dt = rng.choice([0.0025, 0.005])
    leaf = rng.choice([4, 8, 16])
    batch = rng.choice([0, 32, 64])
    width = rng.choice([32, 32, 64])
    fp64 = rng.choice([0, 1, 1])
    if kind == "step":
        return dict(kind=kind, n=_log_int(rng, 1000, 1500000), theta=theta, eps=eps, dt=dt, leaf=leaf, batch=batch,
                    width=width, com_fp64=fp64, graphs=rng.choice([0, 1]))
    if kind == "accels":
        return dict(kind=kind, n=_log_int(rng, 10000, 3000000), theta=theta, eps=eps, leaf=leaf, batch=batch,
                    width=width, com_fp64=fp64)
    if kind == "batched":
        return dict(kind=kind, count=rng.randint(2, 48), n_lo=4096, n_hi=_log_int(rng, 8192, 262144),
                    mix=rng.randint(0, 1 << 20), theta=theta, eps=eps, dt=dt, leaf=leaf, batch=batch, width=width,
                    com_fp64=fp64)
    if kind == "live":
        return dict(kind=kind, n=_log_int(rng, 2000, 1000000))
    if kind == "host":
        return dict(kind=kind, n=_log_int(rng, 2000, 1500000), theta=theta, eps=eps, dt=dt, leaf=leaf, batch=batch,
                    pinned=rng.choice([0, 1]))
    if kind == "served":
        return dict(kind=kind, count=rng.randint(2, 10), n_lo=8192, n_hi=_log_int(rng, 16384, 65536),
                    mix=rng.randint(0, 1 << 20), steps_lo=2, steps_hi=rng.randint(3, 6), slots=rng.randint(2, 6),
                    theta=theta, eps=eps, dt=dt, leaf=leaf, batch=batch)
    if kind == "sort":
        return dict(kind=kind, n=_log_int(rng, 1000, 1048576))
    if kind == "render":
        w, h = rng.choice([(640, 360), (1280, 720), (1920, 1080), (1001, 777)])
        return dict(kind=kind, n=_log_int(rng, 10000, 2000000), w=w, h=h)
    return dict(kind=kind, n=_log_int(rng, 10000, 300000), targets=_log_int(rng, 64, 4096), eps=eps)


# ---- inputs -----------------------------------------------------------------
def _stars(n, seed):
    """The two-galaxy recipe at n particles: the equal pair where n is one of
    the recipe's own sizes, else an unequal pair."""
    for counts in (gcs.SMALL_COUNTS, gcs.LARGE_COUNTS, (512, 128, 64)):
        if n == 2 * sum(counts):
            return gcs.collision_equal(*counts, seed=seed)
    if n == 4194304:  # the precision study's orbit
        return gcs.collision_pair(n, 1.0 / 3.0, 8.0, 0.6, 30.0, seed)
    return gcs.collision_pair(n, 0.6, 6.0, 0.5, 40.0, seed)


def _scenarios(case):
    return workloads.batched_scenarios(case["count"], case["n_lo"], case["n_hi"], seed=case["mix"])


def _scenario_stars(case, seed):
    out = []
    for s in _scenarios(case):
        s.seed = (int(seed) << 8) + s.index
        out.append(s.stars(gcs))
    return out


def _params(case):
    return gcs.reference_params(theta=case["theta"], epsilon_sq=case["eps"] ** 2, dt=case.get("dt", 0.0),
                                leaf_size=case["leaf"], walk_batch=case["batch"], bounds_mode=gcs.BOUNDS_DEVICE,
                                recolor=0, com_fp64=case.get("com_fp64", 1))


_shared = {}


def _stream():
    if "stream" not in _shared:
        _shared["stream"] = torch.cuda.Stream()
    return _shared["stream"].cuda_stream


class _Rows:
    """float4 rows of a context's array; the tensor over them keeps the context alive."""

    def __init__(self, ctx, address):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": (ctx.n, 4), "typestr": "<f4", "data": (address, False), "version": 3}


class _Views:
    """Tensors over a context's current arrays, kept per array (a step alternates between two)."""

    def __init__(self, ctx):
        self.ctx, self.by_address = ctx, {}

    def get(self, which):
        address = self.ctx.device_array(which)
        if address not in self.by_address:
            self.by_address[address] = torch.as_tensor(_Rows(self.ctx, address), device="cuda")
        return self.by_address[address]

    def state(self):
        pos, vel, acc = self.get(gcs.BUF_POS), self.get(gcs.BUF_VEL), self.get(gcs.BUF_ACCEL)
        return {"pos": pos, "vel": vel[:, :3], "tcol": vel.view(torch.int32)[:, 3], "acc": acc[:, :3]}


def _columns(stars):
    """A Star array as plain arrays (views)."""
    return {f: stars[f] for f in stars.dtype.names}


def _pinned_stars(n):
    t = torch.zeros(n * gcs.STAR_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
    return t, t.numpy().view(gcs.STAR_DTYPE)


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind in ("step", "accels", "live", "host", "render", "direct"):
        n = case["n"]
        stars = _stars(n, seed)
        ctx = gcs.Context(n)
        ctx.set_stream(_stream())
        st.update(ctx=ctx, views=_Views(ctx))
        if kind != "host":
            ctx.upload(stars)
        if kind in ("step", "accels"):
            st["p"] = _params(case)
            if kind == "accels":
                st["p"].with_potential = 1
            if case["width"] != 32:
                ctx.set_group_width(case["width"])
            if case.get("graphs"):
                ctx.set_graphs(True)
        elif kind == "live":
            st["p"] = gcs.reference_params()
            st["out"] = np.zeros(n, gcs.STAR_DTYPE)
            st["cols"] = _columns(st["out"])
        elif kind == "host":
            st["p"] = _params(case)
            if case["pinned"]:
                st["keep"], st["in"] = _pinned_stars(n)
                st["keep_out"], st["out"] = _pinned_stars(n)
                st["in"][:] = stars
            else:
                st["in"], st["out"] = stars, np.zeros(n, gcs.STAR_DTYPE)
            st["cols"] = _columns(st["out"])
        elif kind == "render":
            st["cam"], st["w"], st["h"] = _camera(), case["w"], case["h"]
        else:
            st["p"] = gcs.reference_params(epsilon_sq=case["eps"] ** 2)
            st["targets"] = _targets(case, seed)
        return st
    if kind == "batched":
        parts = _scenario_stars(case, seed)
        ctx = gcs.Context(sum(len(s) for s in parts), len(parts))
        ctx.set_stream(_stream())
        ctx.set_segments([len(s) for s in parts])
        ctx.upload(np.concatenate(parts))
        if case["width"] != 32:
            ctx.set_group_width(case["width"])
        ctx.set_graphs(True)
        st.update(ctx=ctx, views=_Views(ctx), p=_params(case))
        return st
    if kind == "served":
        parts = _scenario_stars(case, seed)
        rng = np.random.default_rng(case["mix"])
        steps = [int(x) for x in rng.integers(case["steps_lo"], case["steps_hi"] + 1, len(parts))]
        cap = max(max(len(s) for s in parts), sum(len(s) for s in parts) // 2)
        st.update(parts=parts, steps=steps, srv=gcs.Server(_params(case), cap, case["slots"], 150e9))
        return st
    if kind == "sort":
        n = case["n"]
        keys, vals = _pairs(n, seed)
        st.update(n=n, keys0=keys, vals0=vals, keys=torch.empty_like(keys), vals=torch.empty_like(vals),
                  keys_alt=torch.empty_like(keys), vals_alt=torch.empty_like(vals),
                  status=torch.zeros(1, dtype=torch.int32, device="cuda"))
        return st
    raise ValueError(kind)


def _camera():
    # near enough that both galaxies fill the frame
    cam = gcs.camera_reference()
    cam.pos[:] = (0.0, 20.0, 60.0)
    return gcs.camera_look_at(cam, (0.0, 0.0, 0.0))


def _targets(case, seed):
    return np.sort(np.random.default_rng(seed).choice(case["n"], case["targets"], replace=False)).astype(np.int64)


def _pairs(n, seed):
    """Morton codes of the recipe's particles (what the engine sorts), with
    their positions as values."""
    stars = _stars(n, seed)
    xyz = np.stack([stars["x"], stars["y"], stars["z"]], 1)
    keys = _morton(xyz, xyz.min(), xyz.max())
    return (torch.from_numpy(keys.view(np.int64)).cuda(), torch.arange(n, dtype=torch.int32, device="cuda"))


# ---- one pass -----------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind in ("step", "batched"):
        state["ctx"].step(state["p"])
        return state["views"].state()
    if kind == "accels":
        state["ctx"].compute_accels(state["p"])
        return {"pos": state["views"].get(gcs.BUF_POS), "acc": state["views"].get(gcs.BUF_ACCEL)}
    if kind == "live":
        state["ctx"].step_host(state["p"], state["out"])
        return state["cols"]
    if kind == "host":
        state["ctx"].step_host_io(state["p"], state["in"], state["out"])
        return state["cols"]
    if kind == "render":
        return state["ctx"].render(state["cam"], state["w"], state["h"])
    if kind == "direct":
        return state["ctx"].direct_fp64(state["p"], state["targets"])
    if kind == "served":
        srv, got = state["srv"], {}
        for i, (s, k) in enumerate(zip(state["parts"], state["steps"])):
            srv.submit(i, s, k)
        while len(got) < len(state["parts"]):
            srv.tick()
            r = srv.pop()
            while r is not None:
                got[int(r[0].id)] = r[1]
                r = srv.pop()
        return _columns(np.concatenate([got[i] for i in range(len(state["parts"]))]))
    # the pairs to sort arrive in other buffers, as a caller's encode step leaves them
    state["keys"].copy_(state["keys0"])
    state["vals"].copy_(state["vals0"])
    stream = torch.cuda.current_stream().cuda_stream
    rc = gcs.lib().gcs_sort_pairs_static(state["keys"].data_ptr(), state["vals"].data_ptr(),
                                         state["keys_alt"].data_ptr(), state["vals_alt"].data_ptr(), state["n"],
                                         state["status"].data_ptr(), stream)
    if rc != gcs.OK:
        raise RuntimeError("gcs_sort_pairs_static: %d" % rc)
    return state["keys"], state["vals"]


# ---- what a pass cannot do without ----------------------------------------------
def _terms(n, theta):
    """Walk terms of one particle: about 1,424 at 1,048,576 particles and theta 0.5."""
    return min(float(n), 71.0 * math.log2(max(n, 2)) * (0.5 / theta) ** 2.5)


def work(case):
    kind = case["kind"]
    if kind in ("batched", "served"):
        parts = [s.n for s in _scenarios(case)]
        steps = 1 if kind == "batched" else (case["steps_lo"] + case["steps_hi"]) / 2
        return {"bytes": sum(parts) * (80 if kind == "batched" else 64),
                "flops": sum(steps * n * _terms(n, case["theta"]) * 20 for n in parts)}
    n = case["n"]
    if kind == "sort":
        return {"bytes": 24 * n, "flops": 0}
    if kind == "render":
        return {"bytes": 32 * n + 4 * case["w"] * case["h"], "flops": 100 * n}
    if kind == "direct":
        return {"bytes": 16 * n + 32 * case["targets"], "flops": 20.0 * n * case["targets"]}
    theta = 1.0 if kind == "live" else case["theta"]
    return {"bytes": {"step": 80, "accels": 48, "live": 64, "host": 64}[kind] * n,
            "flops": 20.0 * n * _terms(n, theta)}


def _cost(case):
    w = work(case)
    return max(w["flops"], w["bytes"] * 50.0)


# ---- 64-bit values ---------------------------------------------------------------
def _spread(v):
    x = v.astype(np.uint64) & np.uint64(0x1FFFFF)
    for shift, mask in ((32, 0x001F00000000FFFF), (16, 0x001F0000FF0000FF), (8, 0x100F00F00F00F00F),
                        (4, 0x10C30C30C30C30C3), (2, 0x1249249249249249)):
        x = (x | (x << np.uint64(shift))) & np.uint64(mask)
    return x


def _morton(xyz, lo, hi):
    """63-bit Morton codes in the FP32 arithmetic that defines the sorted order."""
    lo, hi = np.float32(lo), np.float32(hi)
    scale = np.float32(2097151.0) / np.float32(hi - lo)
    q = (xyz.astype(np.float32) - lo) * scale
    q = np.minimum(np.maximum(q, np.float32(0.0)), np.float32(4294967040.0)).astype(np.uint64)
    return (_spread(q[:, 0]) << np.uint64(2)) | (_spread(q[:, 1]) << np.uint64(1)) | _spread(q[:, 2])


def _direct(pos, mass, eps2, targets=None, potential=False):
    """FP64 softened sums over every other particle: [targets, 3] (and potentials)."""
    x = torch.from_numpy(pos.astype(np.float64)).cuda()
    m = torch.from_numpy(mass.astype(np.float64)).cuda()
    idx = torch.arange(len(pos), device="cuda") if targets is None else torch.from_numpy(targets).cuda()
    out = torch.empty(len(idx), 4 if potential else 3, dtype=torch.float64, device="cuda")
    step = max(1, 200_000_000 // len(pos))
    for a in range(0, len(idx), step):
        t = idx[a:a + step]
        d = [x[None, :, k] - x[t][:, None, k] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps2
        inv = r2.rsqrt_()
        inv[torch.arange(len(t), device="cuda"), t] = 0.0
        w = inv * inv * inv * m
        for k in range(3):
            out[a:a + step, k] = (w * d[k]).sum(1)
        if potential:
            out[a:a + step, 3] = -(inv * m).sum(1)
    return out


def _stepped(stars, p):
    """One step of one scenario in 64 bits: (pos with mass, vel, acc), in Morton order."""
    xyz = np.stack([stars["x"], stars["y"], stars["z"]], 1)
    lo, hi = (p.global_min, p.global_max) if p.bounds_mode == gcs.BOUNDS_CALLER else (xyz.min(), xyz.max())
    stars = stars[np.argsort(_morton(xyz, lo, hi), kind="stable")]
    xyz = np.stack([stars["x"], stars["y"], stars["z"]], 1)
    acc = p.G * _direct(xyz, stars["mass"], float(p.epsilon_sq))
    dt = float(p.dt)
    vel = torch.from_numpy(np.stack([stars["vx"], stars["vy"], stars["vz"]], 1).astype(np.float64)).cuda() + acc * dt
    pos = torch.from_numpy(xyz.astype(np.float64)).cuda() + vel * dt
    mass = torch.from_numpy(stars["mass"].astype(np.float64)).cuda()
    return torch.cat([pos, mass[:, None]], 1), vel, acc


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sort", "render", "served"):
        return None  # whole numbers; several steps
    if kind == "direct":
        stars = _stars(case["n"], seed)
        xyz = np.stack([stars["x"], stars["y"], stars["z"]], 1)
        return _direct(xyz, stars["mass"], float(np.float32(case["eps"] ** 2)), _targets(case, seed))
    if kind == "batched":
        parts = _scenario_stars(case, seed)
        if sum(float(len(s)) ** 2 for s in parts) > MAX_PAIRS:
            return None
        p = _params(case)
        got = [torch.cat(x) for x in zip(*(_stepped(s, p) for s in parts))]
        return {"pos": got[0], "vel": got[1], "tcol": None, "acc": got[2]}
    if float(case["n"]) ** 2 > MAX_PAIRS:
        return None
    stars = _stars(case["n"], seed)
    if kind == "accels":
        p = _params(case)
        xyz = np.stack([stars["x"], stars["y"], stars["z"]], 1)
        stars = stars[np.argsort(_morton(xyz, xyz.min(), xyz.max()), kind="stable")]
        xyz = np.stack([stars["x"], stars["y"], stars["z"]], 1)
        pos = torch.from_numpy(np.concatenate([xyz, stars["mass"][:, None]], 1).astype(np.float64))
        return {"pos": pos, "acc": p.G * _direct(xyz, stars["mass"], float(p.epsilon_sq), potential=True)}
    p = gcs.reference_params() if kind == "live" else _params(case)
    pos, vel, acc = _stepped(stars, p)
    if kind == "step":
        return {"pos": pos, "vel": vel, "tcol": None, "acc": acc}
    pos, vel = pos.cpu().numpy(), vel.cpu().numpy()
    out = {"x": pos[:, 0], "y": pos[:, 1], "z": pos[:, 2], "vx": vel[:, 0], "vy": vel[:, 1], "vz": vel[:, 2],
           "mass": pos[:, 3], "type": None, "r": None, "g": None, "b": None}
    return {k: v if v is None else np.ascontiguousarray(v) for k, v in out.items()}
