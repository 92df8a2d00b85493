"""Measured cases: the calls that programs make of this package, over their real range.

Every case goes through the public entry points (``nbodysim_b200.Engine`` and the C ABI behind it). A case is a dict of
plain values; ``kind`` says which call it makes:

  frames    ``step(steps)`` on particles resident on the GPU: the frame loop (one step a frame, or several in one call)
  forces    ``compute_forces()`` on resident particles: the FP64 form that checks and reports use
  dropin    ``barnes_hut(...)`` on host arrays: what replaces the reference's ``barnes_hut_cuda`` call
  ensemble  ``step(steps)`` on many independent systems in one engine
  vjp       ``force_vjp(...)``: the backward of one force pass
  train     ``forward_checkpointed`` + ``backward`` of a loss on the final positions: one training step
  merge     a frame with collisions or the minimum node size, loaded from and read back to the host
  direct    ``direct_forces(targets)``: the all-pairs sums that accuracy reports compare with

Particles come from the seeded generator of the package (cube, sphere, shell), or are a collapsed system: a sphere with
density ~ r^-2 and a few particles thrown far out, which is what the shell turns into after some tens of steps.

Single precision results (the MIXED form computes pair forces in FP32) are handed on as float32, the way a renderer or an
optimiser takes them; the FP64 form's stay float64.
"""
import math

import numpy as np
import torch

import nbodysim_b200 as nb

G = 6.67384e-11
GEN = {"cube": 0, "sphere": 1, "shell": 2}
ADAPTIVE = dict(adaptive=1, min_adaptive_dt=0.00333, max_pos_change=3.0, max_vel_change=3.0)


def listed():
    return [
        # a handful of bodies: one small frame, bounded by launches and the call itself
        {"name": "frame_cube_97", "kind": "frames", "dist": "cube", "n": 97, "theta": 0.5, "steps": 1, "adaptive": False,
         "fp64": False},
        # the small configuration: cube of 5000, one frame of the frame loop (its files are written between frames)
        {"name": "frame_cube_5000", "kind": "frames", "dist": "cube", "n": 5000, "theta": 0.5, "steps": 1,
         "adaptive": False, "fp64": False},
        # the middle configuration: sphere of 100,000, two steps in one call
        {"name": "frames_sphere_100k", "kind": "frames", "dist": "sphere", "n": 100000, "theta": 0.5, "steps": 2,
         "adaptive": False, "fp64": False},
        # the large configuration: shell of 1,048,576 with adaptive dt, one frame
        {"name": "frame_shell_1m", "kind": "frames", "dist": "shell", "n": 1 << 20, "theta": 0.5, "steps": 1,
         "adaptive": True, "fp64": False},
        # the same size once it has collapsed: long lists, deep tree, escaped particles that stretch the root cube
        {"name": "frame_collapsed_1m", "kind": "frames", "dist": "collapsed", "n": 1 << 20, "theta": 0.5, "steps": 1,
         "adaptive": True, "fp64": False},
        # the FP64 form, with damping: forces for a report, an odd size
        {"name": "forces_fp64_sphere_60001", "kind": "forces", "dist": "sphere", "n": 60001, "theta": 0.5, "damping": True,
         "fp64": True},
        # the reference's program with this library linked in (its FLOAT build): host particles in, accelerations out
        {"name": "dropin_float_shell_20011", "kind": "dropin", "dist": "shell", "n": 20011, "theta": 0.5, "damping": False,
         "float_build": True},
        # a batch of systems of uneven size, two steps in one call
        {"name": "ensemble_128", "kind": "ensemble", "systems": 128, "n_min": 1024, "n_max": 16384, "theta": 0.5,
         "steps": 2},
        # the backward of one force pass at the adjoint configuration's size
        {"name": "vjp_sphere_65536", "kind": "vjp", "dist": "sphere", "n": 65536, "theta": 0.5, "damping": False},
        # a training step in the FP64 form: 16 steps with checkpoints, then the reverse pass
        {"name": "train_fp64_sphere_16384", "kind": "train", "dist": "sphere", "n": 16384, "theta": 0.5, "steps": 16,
         "fp64": True},
        # a frame in which particles collide and merge, from host arrays and back
        {"name": "merge_cube_60000", "kind": "merge", "dist": "cube", "n": 60000, "theta": 0.5, "collision_range": 0.5,
         "min_node_size": 0.0},
        # the accuracy report of the middle configuration: 4096 targets against all particles
        {"name": "direct_sphere_100k", "kind": "direct", "dist": "sphere", "n": 100000, "targets": 4096, "damping": False},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["frames", "frames", "frames", "frames", "forces", "dropin", "dropin", "ensemble", "vjp", "train",
                       "merge", "direct"])
    dist = rng.choice(["cube", "sphere", "shell", "collapsed"])
    theta = rng.choice([0.4, 0.5, 0.5, 0.7])
    if kind == "frames":
        n = _log_int(rng, 64, 1 << 20)
        steps = rng.choice([1, 1, 1, 2]) if n <= 300000 else 1
        return {"kind": kind, "dist": dist, "n": n, "theta": theta if n <= 300000 else max(theta, 0.5), "steps": steps,
                "adaptive": steps == 1 and rng.random() < 0.5, "fp64": n <= 100000 and rng.random() < 0.25}
    if kind == "forces":
        return {"kind": kind, "dist": dist, "n": _log_int(rng, 64, 100000), "theta": theta,
                "damping": rng.random() < 0.5, "fp64": rng.random() < 0.7}
    if kind == "dropin":
        return {"kind": kind, "dist": rng.choice(["cube", "sphere", "shell"]), "n": _log_int(rng, 64, 100000),
                "theta": theta, "damping": rng.random() < 0.3, "float_build": rng.random() < 0.5}
    if kind == "ensemble":
        return {"kind": kind, "systems": _log_int(rng, 3, 150), "n_min": rng.choice([33, 200, 1024]),
                "n_max": _log_int(rng, 2000, 16384), "theta": theta, "steps": rng.choice([1, 2])}
    if kind == "vjp":
        return {"kind": kind, "dist": rng.choice(["cube", "sphere", "shell"]), "n": _log_int(rng, 64, 65536),
                "theta": theta, "damping": rng.random() < 0.3}
    if kind == "train":
        return {"kind": kind, "dist": rng.choice(["cube", "sphere", "shell"]), "n": _log_int(rng, 64, 12000),
                "theta": max(theta, 0.5), "steps": rng.randint(2, 16), "fp64": rng.random() < 0.7}
    if kind == "merge":
        return {"kind": kind, "dist": "cube", "n": _log_int(rng, 1000, 60000), "theta": theta,
                "collision_range": rng.uniform(0.2, 1.0), "min_node_size": rng.choice([0.0, 0.0, 2.0])}
    return {"kind": kind, "dist": rng.choice(["cube", "sphere", "shell"]), "n": _log_int(rng, 1000, 100000),
            "targets": rng.randint(100, 4096), "damping": rng.random() < 0.3}


# ---- inputs ------------------------------------------------------------------------------------------------------------


def _particles(dist, n, seed):
    """Host particles (pos, vel, mass) of the named distribution."""
    seed = 1 + (int(seed) * 2654435761 + 12345) % 2147483000
    if dist == "collapsed":
        rng = np.random.default_rng(seed)
        r = 100.0 * rng.uniform(0.0, 1.0, n)
        far = n // 1000
        r[:far] = 100.0 * np.exp(rng.uniform(0.0, math.log(1e4), far))
        d = rng.normal(size=(n, 3))
        d /= np.linalg.norm(d, axis=1)[:, None]
        order = rng.permutation(n)
        pos = np.ascontiguousarray((d * r[:, None])[order])
        return pos, 30.0 * rng.normal(size=(n, 3)), rng.uniform(5e10, 5e11, n)
    size = {"cube": 512.0, "sphere": 512.0, "shell": 1024.0}[dist]
    return nb.generate(n, gen_type=GEN[dist], size=size, r_sphere=100.0, rotation_magnitude=0.1, seed=seed)


def _system_sizes(case):
    rng = np.random.default_rng(case["systems"])
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    return np.exp(rng.uniform(lo, hi, case["systems"])).astype(np.uint32)


def _systems(case, seed):
    counts = _system_sizes(case)
    parts = [_particles(("cube", "sphere", "shell")[k % 3], int(c), 1000 * int(seed) + k) for k, c in enumerate(counts)]
    return counts, [np.concatenate([p[q] for p in parts]) for q in range(3)]


class _View:
    """An engine buffer on the GPU as torch takes it; a tensor made of it keeps the engine, which owns the memory."""

    def __init__(self, eng, ptr, shape, typestr):
        self.eng = eng
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _resident(eng):
    """The engine's positions, velocities and accelerations as tensors over its own memory."""
    v = eng.device_view()
    at = [(v.pos, "<f8"), (v.vel, "<f8"), (v.acc, "<f8" if v.acc_is_double else "<f4")]
    return [torch.as_tensor(_View(eng, p, (v.n, 3), t), device="cuda") for p, t in at]


def _own_stream(eng):
    """Engine and torch work on one stream, as in a program that uses both."""
    s = torch.cuda.Stream()
    nb.load_library().nbody_set_stream(eng._h, s.cuda_stream)
    return s


def _precision(case):
    return nb.PRECISION_FP64 if case.get("fp64") else nb.PRECISION_MIXED


def _step_params(case):
    # calls of several steps take a fine step: unsoftened close pairs would otherwise blow rounding up from step to step
    kind = case["kind"]
    if kind == "train":
        return dict(dt=0.001)
    if kind == "ensemble" or case.get("steps", 1) > 1:
        return dict(dt=0.0005)
    return dict(ADAPTIVE) if case.get("adaptive") else {}


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "ensemble":
        counts, (pos, vel, mass) = _systems(case, seed)
    else:
        pos, vel, mass = _particles(case["dist"], case["n"], seed)
    if kind in ("frames", "ensemble", "forces"):
        eng = nb.Engine(theta=case["theta"], damping=int(case.get("damping", False)), precision=_precision(case),
                        **_step_params(case))
        st["stream"] = _own_stream(eng)
        if kind == "ensemble":
            eng.set_systems(counts)
        eng.set_particles(pos, vel, mass)
        st["views"] = _resident(eng)
        st["pos0"], st["vel0"] = torch.from_numpy(pos).cuda(), torch.from_numpy(vel).cuda()
    elif kind == "dropin":
        eng = nb.Engine(datatype_bytes=4 if case["float_build"] else 8)
    elif kind == "vjp":
        eng = nb.Engine(theta=case["theta"], damping=int(case["damping"]))
        st["cot"] = np.random.default_rng(int(seed)).normal(size=pos.shape)
    elif kind == "train":
        eng = nb.Engine(theta=case["theta"], precision=_precision(case), **_step_params(case))
        st["target"] = pos + np.random.default_rng(int(seed)).normal(0.0, 5.0, pos.shape)
    elif kind == "merge":
        eng = nb.Engine(theta=case["theta"], collide=1, collision_range=case["collision_range"],
                        min_node_size=case["min_node_size"])
    else:
        eng = nb.Engine()
        eng.set_particles(pos, vel, mass)
        rng = np.random.default_rng(int(seed))
        st["targets"] = np.sort(rng.choice(case["n"], min(case["targets"], case["n"]), replace=False)).astype(np.uint32)
    torch.cuda.synchronize()
    st.update(eng=eng, pos=pos, vel=vel, mass=mass)
    return st


# ---- one pass ----------------------------------------------------------------------------------------------------------


def run(st):
    case, eng = st["case"], st["eng"]
    kind = case["kind"]
    if kind in ("frames", "ensemble"):
        pos, vel, acc = st["views"]
        with torch.cuda.stream(st["stream"]):
            pos.copy_(st["pos0"])
            vel.copy_(st["vel0"])
            eng.step(case["steps"])
            if case.get("fp64"):
                return {"pos": pos, "vel": vel, "acc": acc}
            return {"pos": pos.float(), "vel": vel.float(), "acc": acc}
    if kind == "forces":
        eng.compute_forces()
        return {"acc": st["views"][2]}
    if kind == "dropin":
        acc, counts = eng.barnes_hut(st["pos"], st["mass"], damping=case["damping"], theta=case["theta"], counts=True)
        return {"acc": acc.astype(np.float32), "counts": counts}
    if kind == "vjp":
        gp, gm = eng.force_vjp(st["pos"], st["mass"], st["cot"])
        return {"dpos": gp.astype(np.float32), "dmass": gm.astype(np.float32)}
    if kind == "train":
        eng.set_particles(st["pos"], st["vel"], st["mass"])
        eng.forward_checkpointed(case["steps"])
        x, v = eng.get_particles()
        got = eng.backward(2.0 * (x - st["target"]) / case["n"])
        names = ("x", "v", "dpos", "dvel", "dmass")
        return {k: a if case["fp64"] else a.astype(np.float32) for k, a in zip(names, (x, v) + tuple(got))}
    if kind == "merge":
        eng.set_particles(st["pos"], st["vel"], st["mass"])
        eng.step(1)
        x, v = eng.get_particles()
        out = {"pos": np.zeros((case["n"], 3), np.float32), "vel": np.zeros((case["n"], 3), np.float32),
               "mass": np.zeros(case["n"])}  # room for every particle; the merged ones leave zeros at the end
        for name, a in (("pos", x), ("vel", v), ("mass", eng.get_masses())):
            out[name][:len(a)] = a
        return out
    return {"acc": eng.direct_forces(st["targets"], damping=case["damping"])}


# ---- what a pass cannot do without -------------------------------------------------------------------------------------

# Accepted nodes per particle at theta 0.5: a + b log2 n, fitted to the reference's counts between 1000 and 1,048,576.
_COUNTS = {"cube": (-480.0, 67.0), "sphere": (-560.0, 78.0), "shell": (-140.0, 27.0), "collapsed": (-1100.0, 158.0)}


def _interactions(dist, n, theta):
    a, b = _COUNTS[dist]
    return n * min(n - 1.0, max(a + b * math.log2(n), 20.0 + 10.0 * math.log2(n)) * (0.5 / theta) ** 1.8)


def work(case):
    """Bytes: each input once, each output once. Flops: 20 per accepted particle-node pair (the customary count)."""
    kind = case["kind"]
    if kind == "direct":
        m = min(case["targets"], case["n"])
        return {"bytes": 32.0 * case["n"] + 28.0 * m, "flops": 20.0 * m * case["n"]}
    if kind == "ensemble":
        lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
        n = case["systems"] * (case["n_max"] - case["n_min"]) / max(hi - lo, 1e-9)
        pairs = case["systems"] * _interactions("sphere", n / case["systems"], case["theta"])
        steps = case["steps"]
    else:
        n, steps = case["n"], case.get("steps", 1)
        pairs = _interactions(case["dist"], n, case["theta"])
    if kind in ("frames", "ensemble"):
        return {"bytes": n * (steps * (56.0 + 48.0 + 12.0) + 96.0), "flops": 20.0 * pairs * steps}
    if kind == "forces":
        return {"bytes": n * (32.0 + 24.0), "flops": 20.0 * pairs}
    if kind == "dropin":
        return {"bytes": n * (32.0 + 28.0), "flops": 20.0 * pairs}
    if kind == "vjp":
        return {"bytes": n * (56.0 + 32.0), "flops": 60.0 * pairs}
    if kind == "train":
        return {"bytes": n * steps * 3 * 104.0, "flops": (20.0 + 20.0 + 60.0) * pairs * steps}
    return {"bytes": n * (56.0 + 56.0), "flops": 20.0 * pairs}


# ---- the same results in 64 bits, in plain torch -----------------------------------------------------------------------


class _Octree:
    """The reference's octree, level by level: cells of the root cube that hold particles, split while they hold two."""

    def __init__(self, pos, mass):
        n = len(mass)
        lo, hi = pos.min(0).values, pos.max(0).values
        e = [float(v) for v in hi - lo]
        side = e[0] if e[0] > e[1] and e[0] > e[2] else e[1] if e[1] > e[0] and e[1] > e[2] else e[2]
        self.pos, self.mass, self.levels = pos, mass, []
        who = torch.arange(n, device=pos.device)
        cell = torch.zeros(n, dtype=torch.int64, device=pos.device)
        centre = ((lo + hi) / 2.0).expand(n, 3).clone()
        side, cells = side + 2.0, 1
        while len(who):
            count = torch.bincount(cell, minlength=cells)
            m = torch.zeros(cells, dtype=torch.float64, device=pos.device).index_add_(0, cell, mass[who])
            com = torch.zeros(cells, 3, dtype=torch.float64, device=pos.device)
            com.index_add_(0, cell, pos[who] * mass[who][:, None])
            com /= m[:, None]
            leaf = torch.full((cells,), -1, dtype=torch.int64, device=pos.device)
            one = count[cell] == 1
            leaf[cell[one]] = who[one]
            com[cell[one]] = pos[who[one]]
            lv = {"side": side, "com": com, "mass": m, "leaf": leaf, "who": who, "cell": cell,
                  "first": torch.zeros(cells, dtype=torch.int64, device=pos.device),
                  "children": torch.zeros(cells, dtype=torch.int64, device=pos.device)}
            self.levels.append(lv)
            who, cell, centre = who[~one], cell[~one], centre[~one]
            if not len(who):
                break
            up = pos[who] > centre
            half = side / 2.0
            centre = centre + (2.0 * up.double() - 1.0) * (half / 2.0)
            digit = up[:, 0].long() + 2 * up[:, 1].long() + 4 * up[:, 2].long()
            keys, cell = torch.unique(cell * 8 + digit, return_inverse=True)
            cells, side = len(keys), half
            parent = keys // 8
            lv["children"] = torch.bincount(parent, minlength=len(leaf))
            lv["first"] = torch.cumsum(lv["children"], 0) - lv["children"]

    def pairs(self, theta, chunk):
        """Accepted (level, particle, node), for `chunk` particles at a time; particles ascend."""
        n = len(self.mass)
        for a in range(0, n, chunk):
            p = torch.arange(a, min(n, a + chunk), device=self.pos.device)
            node = torch.zeros_like(p)
            for lv in self.levels:
                d = lv["com"][node] - self.pos[p]
                dist = torch.sqrt(d[:, 0] ** 2 + d[:, 1] ** 2 + d[:, 2] ** 2)
                inner = lv["leaf"][node] < 0
                opened = inner & (lv["side"] / dist > theta)
                take = ~opened & (lv["leaf"][node] != p)
                yield a, min(n, a + chunk), lv, p[take], node[take], d[take], dist[take]
                p, node = p[opened], node[opened]
                if not len(p):
                    break
                k = lv["children"][node]
                p = torch.repeat_interleave(p, k)
                base = torch.repeat_interleave(lv["first"][node] - (torch.cumsum(k, 0) - k), k)
                node = base + torch.arange(len(p), device=p.device)


def _chunk(n):
    return max(64, min(n, 1 << 16))


def _exact_forces(pos, mass, theta, damping=False):
    acc = torch.zeros_like(pos)
    for a, b, lv, p, node, d, r in _Octree(pos, mass).pairs(theta, _chunk(len(mass))):
        den = r * r + torch.exp(-r) if damping else r * r
        f = (G * lv["mass"][node] / (den * r))[:, None] * d
        lengths = torch.bincount(p - a, minlength=b - a)
        acc[a:b] += torch.segment_reduce(f, "sum", lengths=lengths, axis=0, initial=0.0)
    return acc


def _exact_vjp(pos, mass, lam, theta, damping=False):
    """(dL/dpos, dL/dmass) of the forces with frozen opening decisions, for the cotangents lam = dL/dacc."""
    tree = _Octree(pos, mass)
    gx, gm = torch.zeros_like(pos), torch.zeros_like(mass)
    adj = [torch.zeros(len(lv["mass"]), 4, dtype=torch.float64, device=pos.device) for lv in tree.levels]
    at = {id(lv): k for k, lv in enumerate(tree.levels)}
    for a, b, lv, p, node, d, r in tree.pairs(theta, _chunk(len(mass))):
        if damping:
            ex = torch.exp(-r)
            den = r * r + ex
            g, h = 1.0 / (r * den), -(3.0 * r * r + ex - r * ex) / (r ** 3 * den * den)
        else:
            g, h = r ** -3.0, -3.0 * r ** -5.0
        la = lam[p]
        s = (d * la).sum(1)
        v = (G * lv["mass"][node])[:, None] * (g[:, None] * la + (h * s)[:, None] * d)
        gx.index_add_(0, p, -v)
        adj[at[id(lv)]].index_add_(0, node, torch.cat([v, (G * g * s)[:, None]], 1))
    for lv, an in zip(tree.levels, adj):
        who, cell = lv["who"], lv["cell"]
        m, c, q = lv["mass"][cell], lv["com"][cell], an[cell]
        gx[who] += (mass[who] / m)[:, None] * q[:, :3]
        gm[who] += ((pos[who] - c) * q[:, :3]).sum(1) / m + q[:, 3]
    return gx, gm


def _exact_step(pos, vel, mass, theta, dt, adaptive, damping=False):
    acc = _exact_forces(pos, mass, theta, damping)
    if adaptive:
        amax, vmax = float(acc.norm(dim=1).max()), float(vel.norm(dim=1).max())
        lim = dt
        if amax > 0:
            lim = min(lim, ADAPTIVE["max_vel_change"] / amax)
        if vmax > 0:
            lim = min(lim, ADAPTIVE["max_pos_change"] / vmax)
        dt = min(max(lim, ADAPTIVE["min_adaptive_dt"]), dt)
    vel = vel + acc * dt
    return pos + vel * dt, vel, acc


def _exact_train(case, pos, vel, mass, target):
    theta, dt, xs = case["theta"], _step_params(case)["dt"], []
    x, v = pos, vel
    for _ in range(case["steps"]):
        xs.append(x)
        x, v, _ = _exact_step(x, v, mass, theta, dt, False)
    lx, lv, lm = 2.0 * (x - target) / case["n"], torch.zeros_like(vel), torch.zeros_like(mass)
    for xk in reversed(xs):
        lv = lv + lx * dt
        gx, gm = _exact_vjp(xk, mass, lv * dt, theta)
        lx, lm = lx + gx, lm + gm
    return {"x": x, "v": v, "dpos": lx, "dvel": lv, "dmass": lm}


def _exact_direct(pos, mass, targets, damping):
    out = torch.zeros(len(targets), 3, dtype=torch.float64, device=pos.device)
    for a in range(0, len(targets), 256):
        t = targets[a:a + 256]
        d = pos[None] - pos[t][:, None]
        r = torch.sqrt((d * d).sum(2))
        den = r * r + torch.exp(-r) if damping else r * r
        f = G * mass[None] / (den * r)
        f[torch.arange(len(t), device=f.device), t] = 0.0
        out[a:a + 256] = (f[:, :, None] * d).sum(1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "merge" or case.get("float_build"):
        return None  # merged in another order of particles; decisions in float
    if kind == "ensemble":
        counts, arrays = _systems(case, seed)
    else:
        arrays = _particles(case["dist"], case["n"], seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    pos, vel, mass = (torch.from_numpy(a).to(dev) for a in arrays)
    if kind == "direct":
        rng = np.random.default_rng(int(seed))
        t = np.sort(rng.choice(case["n"], min(case["targets"], case["n"]), replace=False)).astype(np.int64)
        return {"acc": _exact_direct(pos, mass, torch.from_numpy(t).to(dev), case["damping"])}
    if kind == "forces":
        return {"acc": _exact_forces(pos, mass, case["theta"], case["damping"])}
    if kind == "dropin":
        return {"acc": _exact_forces(pos, mass, case["theta"], case["damping"]), "counts": None}
    if kind == "vjp":
        cot = torch.from_numpy(np.random.default_rng(int(seed)).normal(size=tuple(pos.shape))).to(dev)
        gx, gm = _exact_vjp(pos, mass, cot, case["theta"], case["damping"])
        return {"dpos": gx, "dmass": gm}
    if kind == "train":
        target = pos + torch.from_numpy(np.random.default_rng(int(seed)).normal(0.0, 5.0, tuple(pos.shape))).to(dev)
        return _exact_train(case, pos, vel, mass, target)
    dt = _step_params(case).get("dt", 0.0333)
    ends = np.cumsum(counts.astype(np.int64)) if kind == "ensemble" else [case["n"]]
    out, a = [], 0
    for b in ends:
        x, v, m = pos[a:b], vel[a:b], mass[a:b]
        for _ in range(case["steps"]):
            x, v, acc = _exact_step(x, v, m, case["theta"], dt, case.get("adaptive", False))
        out.append((x, v, acc))
        a = b
    return {k: torch.cat([o[q] for o in out]) for q, k in enumerate(("pos", "vel", "acc"))}
