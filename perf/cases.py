"""The performance cases of the framework: worlds stepped, rolled out and
differentiated through ``blobs_gb300.native``, the collision-event stream and
the spatial hash, over the sizes these are used at.

A pass over a world goes back to a kept state (``World.restore``, as an
episode or a planning rollout does), steps from it and reads the bodies into
pinned host memory; every pass of a state therefore does the same work and
gives the same results.  The kept state is one step into the scene, past the
velocity requests of a fresh world; the differentiable rollouts start at the
scene itself, because those requests are their parameters.

``exact`` evaluates the same scenes in float64 with torch.  Contact dynamics
amplify rounding: where the float32 and float64 trajectories have parted
(velocities of crowded worlds, gradients over many steps) there is no such
value.
"""
import math

import numpy as np
import torch

from blobs_gb300 import native, scenes

# Upper ends of the drawn sizes: the largest listed case of each kind.
MAX_BODY_STEPS = 4_000_000


def listed():
    return [
        # One frame of a game: the 1,000-sphere walled scene, a step and a read per frame.
        {"name": "frame_1k", "kind": "spheres", "n": 1000, "packing": 0.079, "rmin": 0.1, "rmax": 0.3, "hz": 60,
         "steps": 1, "springs": 0.0, "statics": 0.0},
        # One frame of a larger game that listens to its collisions (the C++ mirror always does): springs,
        # static bodies, a step, the frame's events in order, and a read.
        {"name": "frame_events_20k", "kind": "events", "n": 20_011, "packing": 0.5, "rmin": 0.05, "rmax": 0.15,
         "hz": 60, "steps": 1, "springs": 0.1, "statics": 0.02},
        # An ordinary headless rollout: a pile of a hundred thousand spheres.
        {"name": "rollout_120k", "kind": "spheres", "n": 120_001, "packing": 0.6, "rmin": 0.05, "rmax": 0.15,
         "hz": 120, "steps": 8, "springs": 0.0, "statics": 0.0},
        # The benchmark's world: 1M spheres at 40% packing.
        {"name": "spheres_1m", "kind": "spheres", "n": 1_000_000, "packing": 0.4, "rmin": 0.05, "rmax": 0.15,
         "hz": 120, "steps": 4, "springs": 0.0, "statics": 0.0},
        # The same world at the density that its rollout settles to.
        {"name": "pile_1m", "kind": "spheres", "n": 1_000_000, "packing": 0.8, "rmin": 0.05, "rmax": 0.15,
         "hz": 120, "steps": 4, "springs": 0.0, "statics": 0.0},
        # The same spheres spread over the literal 2000 x 2000 box: few contacts, many empty cells.
        {"name": "sparse_1m", "kind": "spheres", "n": 1_000_000, "packing": 0.0085, "rmin": 0.05, "rmax": 0.15,
         "hz": 120, "steps": 4, "springs": 0.0, "statics": 0.0},
        # One frame of jointed, sprung multi-collider bodies at a game's size.
        {"name": "frame_jointed_2k", "kind": "jointed", "n": 2003, "hz": 120, "steps": 1},
        # The structured world of the benchmark: 200k bodies, ~500k colliders, 50k joints, 100k springs.
        {"name": "jointed_200k", "kind": "jointed", "n": 200_000, "hz": 120, "steps": 4},
        # A training batch of uneven worlds, body counts log-uniform in [64, 8192], every one stepped in one launch.
        {"name": "batch_1024", "kind": "batch", "worlds": 1024, "nmin": 64, "nmax": 8192, "hz": 60, "steps": 4},
        # A small differentiable batch over a short horizon with two checkpoints.
        {"name": "gradient_16x512", "kind": "gradient", "worlds": 16, "n": 512, "hz": 60, "steps": 2, "every": 1},
        # The differentiable batch of the benchmark over one checkpoint segment: recorded forward and backward.
        {"name": "gradient_256x2048", "kind": "gradient", "worlds": 256, "n": 2048, "hz": 60, "steps": 16, "every": 16},
        # SpatialHash: a frame's points inserted and neighbours looked up for a quarter of them.
        {"name": "hash_100k", "kind": "hash", "n": 100_003, "queries": 25_001},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spheres", "spheres", "spheres", "events", "jointed", "jointed", "batch", "batch", "gradient",
                       "hash"])
    if kind in ("spheres", "events"):
        n = _log_int(rng, 300, 1_000_000 if kind == "spheres" else 30_000)
        big = rng.random() < 0.5
        case = {"kind": kind, "n": n,
                "packing": math.exp(rng.uniform(math.log(0.0085), math.log(0.2))) if rng.random() < 0.25
                else rng.uniform(0.2, 0.8),
                "rmin": 0.1 if big else 0.05, "rmax": 0.3 if big else 0.15, "hz": rng.choice([60, 120]),
                "steps": rng.randint(1, max(1, min(10, MAX_BODY_STEPS // n))) if kind == "spheres" else 1,
                "springs": rng.choice([0.0, 0.0, 0.1, 0.5]), "statics": rng.choice([0.0, 0.0, 0.02])}
        if kind == "spheres" and n > 300_000:  # the largest worlds are plain spheres
            case["springs"] = case["statics"] = 0.0
        return case
    if kind == "jointed":
        n = _log_int(rng, 300, 200_000)
        return {"kind": kind, "n": n, "hz": rng.choice([60, 120]), "steps": rng.randint(1, 4)}
    if kind == "batch":
        worlds = _log_int(rng, 8, 1024)
        nmax = _log_int(rng, 128, 8192)
        return {"kind": kind, "worlds": worlds, "nmin": min(64, nmax // 2), "nmax": nmax, "hz": rng.choice([60, 120]),
                "steps": rng.randint(1, 4)}
    if kind == "gradient":
        steps = rng.randint(2, 16)
        return {"kind": kind, "worlds": _log_int(rng, 4, 256), "n": _log_int(rng, 100, 2048), "hz": 60,
                "steps": steps, "every": rng.randint(max(1, steps // 4), steps)}
    n = _log_int(rng, 1000, 100_003)
    return {"kind": "hash", "n": n, "queries": max(1, int(n * rng.uniform(0.05, 0.25)))}


# ---- scenes --------------------------------------------------------------------

def _spheres(case, rng, counts, packing, rmin, rmax, sigma):
    """Worlds of counts[w] overlapping spheres at uniform places in walled
    square boxes, packed back to back."""
    counts = np.asarray(counts, np.int64)
    n = int(counts.sum())
    half = np.array([scenes.box_side(int(c), rmin, rmax, packing) / 2.0 for c in counts], np.float32)
    h = np.repeat(half, counts)[:, None]
    rad = rng.uniform(rmin, rmax, n).astype(np.float32)
    pos = (rng.uniform(-1.0, 1.0, (n, 2)).astype(np.float32) * h).astype(np.float32)
    pos = np.clip(pos, -h + rad[:, None], h - rad[:, None]).astype(np.float32)
    vel = rng.normal(0.0, sigma, (n, 2)).astype(np.float32)
    s = scenes.spheres(pos, rad, vel)
    s.world_box = np.stack([-half, -half, half, half], 1).astype(np.float32)
    if len(counts) > 1:
        off = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)
        s.world_body_offsets, s.world_collider_offsets = off, off.copy()
        s.world_spring_offsets = np.zeros(len(counts) + 1, np.uint32)
        s.world_joint_offsets = np.zeros(len(counts) + 1, np.uint32)
    s.dt = 1.0 / case["hz"]
    return s


def _springs(s, rng, counts, per_world, k_range, c_range, reach):
    """per_world[w] springs in world w, each between bodies next to each other
    in strips of height `reach` (rest = initial distance)."""
    counts = np.asarray(counts, np.int64)
    world = np.repeat(np.arange(len(counts)), counts)
    strip = np.floor(s.pos[:, 1] / reach).astype(np.int64)
    order = np.lexsort((s.pos[:, 0], strip, world))
    start = np.concatenate([[0], np.cumsum(counts)])
    a, b, off = [], [], [0]
    for w, m in enumerate(per_world):
        at = start[w] + rng.choice(int(counts[w]) - 1, size=min(int(m), int(counts[w]) - 1), replace=False)
        a.append(order[at])
        b.append(order[at + 1])
        off.append(off[-1] + len(at))
    a, b = np.concatenate(a), np.concatenate(b)
    k = np.exp(rng.uniform(math.log(k_range[0]), math.log(k_range[1]), len(a))).astype(np.float32)
    c = rng.uniform(c_range[0], c_range[1], len(a)).astype(np.float32)
    scenes.add_springs(s, np.minimum(a, b), np.maximum(a, b), k, c)
    if len(counts) > 1:
        s.world_spring_offsets = np.asarray(off, np.uint32)


def _scene(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    kind = case["kind"]
    if kind in ("spheres", "events"):
        n = case["n"]
        s = _spheres(case, rng, [n], case["packing"], case["rmin"], case["rmax"], 0.5)
        if case["statics"]:
            s.body_type = (rng.random(n) < case["statics"]).astype(np.uint8)
        if case["springs"]:
            _springs(s, rng, [n], [max(1, int(case["springs"] * n))], (200.0, 200.0), (1.0, 1.0), 2 * case["rmax"])
        return s
    if kind == "jointed":
        # the structured world's density: 200k bodies in a 1500 x 1500 box
        n = case["n"]
        s = scenes.jointed_bodies(seed=seed, n=n, n_joints=n // 4, n_springs=n // 2,
                                  side=1500.0 * math.sqrt(n / 200_000))
        s.dt = 1.0 / case["hz"]
        return s
    if kind == "batch":
        counts = np.exp(np.linspace(math.log(case["nmin"]), math.log(case["nmax"]), case["worlds"])).round()
        counts = np.random.Generator(np.random.PCG64(case["worlds"])).permutation(counts.astype(np.int64))
        s = _spheres(case, rng, counts, 0.35, 0.1, 0.3, 1.0)
        _springs(s, rng, counts, np.maximum(1, counts // 10), (200.0, 200.0), (1.0, 1.0), 0.6)
        return s
    counts = [case["n"]] * case["worlds"]
    s = _spheres(case, rng, counts, 0.30, 0.1, 0.2, 1.0)
    _springs(s, rng, counts, [case["n"] // 2] * case["worlds"], (100.0, 5000.0), (0.0, 0.0), 0.4)
    return s


def _targets(case, seed, scene):
    """64 marked bodies per world (fewer in small worlds) and their targets."""
    rng = np.random.Generator(np.random.PCG64([seed, 1]))
    n, m = case["n"], min(64, case["n"] // 2)
    marked = np.concatenate([w * n + rng.choice(n, size=m, replace=False) for w in range(case["worlds"])])
    target = scene.pos[marked] + rng.normal(0.0, 1.0, (len(marked), 2)).astype(np.float32)
    return marked, target.astype(np.float32)


def _points(case, seed):
    """Points and queries of the spatial hash: unique ids, ~10 neighbours a query, cells of 0.6."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n, q = case["n"], case["queries"]
    side = math.sqrt(n / 12.0)
    ids = rng.permutation(4 * n)[:n].astype(np.uint64)
    xy = rng.uniform(-side, side, (n, 2)).astype(np.float32)
    radius = rng.uniform(0.05, 0.15, n).astype(np.float32)
    return ids, xy, radius, xy[rng.choice(n, size=q, replace=False)].copy(), np.full(q, 0.5, np.float32)


# ---- the passes ----------------------------------------------------------------

def _pinned(*shape):
    return torch.empty(*shape, dtype=torch.float32, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "hash":
        ids, xy, radius, qxy, qr = _points(case, seed)
        return {"case": case, "hash": native.SpatialHash(0.6), "ids": ids, "xy": xy, "radius": radius, "qxy": qxy,
                "qr": qr, "found": np.zeros(48 * case["queries"], np.int64)}
    s = _scene(case, seed)
    n = s.n_bodies
    w = native.World(s)
    st = {"case": case, "world": w, "dt": s.dt, "pos": _pinned(n, 2), "pos_old": _pinned(n, 2), "vel": _pinned(n, 2)}
    if kind == "jointed":
        st["rotation"] = _pinned(n)
    if kind == "gradient":
        st["marked"], st["target"] = _targets(case, seed, s)
        st["n_springs"] = s.n_springs
        st["g"] = np.zeros((n, 2), np.float32)
    else:
        if kind == "events":
            w.set_events(True, capacity=64 * n)
            m = 24 * n  # the program's own buffers for a frame's events
            st["events"] = {"a": np.zeros(m, np.int32), "b": np.zeros(m, np.int32),
                            "va": np.zeros((m, 2), np.float32), "vb": np.zeros((m, 2), np.float32)}
        w.step(s.dt)
        if kind == "events":
            w.drain_events()
    w.snapshot()
    w.sync()
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "hash":
        h = state["hash"]
        h.set_points(state["ids"], state["xy"], state["radius"])
        offsets, ids = h.query(state["qxy"], state["qr"])
        state["found"][:len(ids)] = ids.view(np.int64)
        return {"offsets": offsets.view(np.int64), "ids": state["found"]}
    w = state["world"]
    w.restore()
    if kind == "gradient":
        w.rollout_record(state["dt"], case["steps"], case["every"])
        w.read_bodies_into(pos=state["pos"])
        g, m = state["g"], state["marked"]
        g[m] = (state["pos"][m] - state["target"]) * np.float32(2.0 / len(m))
        dv, dk = w.backward(g, state["n_springs"])
        return {"pos": state["pos"], "dv": dv, "dk": dk}
    if case["steps"] == 1:
        w.step(state["dt"])
    else:
        w.rollout(state["dt"], case["steps"])
    out = {"pos": state["pos"], "pos_old": state["pos_old"], "vel": state["vel"]}
    if kind == "events":
        a, b, va, vb = w.drain_events()
        for k, v in (("a", a.view(np.int32)), ("b", b.view(np.int32)), ("va", va), ("vb", vb)):
            state["events"][k][:len(v)] = v
        out["n_events"] = len(a)
        out.update(state["events"])
    if kind == "jointed":
        out["rotation"] = state["rotation"]
    w.read_bodies_into(pos=state["pos"], pos_old=state["pos_old"], vel=state["vel"],
                       rotation=state.get("rotation"))
    return out


def work(case):
    """State read and results written once; ~10 candidate tests and ~2
    contacts per collider in each of a step's 8 substeps."""
    kind = case["kind"]
    if kind == "hash":
        return {"bytes": 20.0 * case["n"] + 20.0 * case["queries"] + 80.0 * case["queries"],
                "flops": 8.0 * 40.0 * case["queries"]}
    if kind == "batch":
        lo, hi = case["nmin"], case["nmax"]
        n = case["worlds"] * (hi - lo) / math.log(hi / lo)
    else:
        n = case["n"] * case.get("worlds", 1)
    sub = 8.0 * case["steps"] * n
    if kind == "jointed":
        # per body 2.5 colliders, half a spring, a quarter of a joint swept four times a substep
        return {"bytes": (28.0 + 28.0 + 2.5 * 24.0 + 0.5 * 20.0 + 0.25 * 40.0) * n, "flops": 700.0 * sub}
    if kind == "gradient":
        # forward, recomputation and reverse; the state of one segment's substeps kept
        return {"bytes": (32.0 + 16.0 + 8.0 + 0.5 * 24.0) * n + 16.0 * 8.0 * case["every"] * n, "flops": 600.0 * sub}
    flops = 40.0 + 100.0 * min(1.0, case.get("packing", 0.35) + 0.1)
    return {"bytes": (32.0 + 24.0) * n + (32.0 * n if kind == "events" else 0.0), "flops": flops * sub}


# ---- the same in float64 -------------------------------------------------------

class _Exact:
    """The reference's substep loop on a whole scene, in float64."""

    def __init__(self, s):
        self.dev = dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")

        def f(a):
            return torch.from_numpy(np.array(a, np.float64)).to(dev)

        def i(a):
            return torch.from_numpy(np.array(a, np.int64)).to(dev)

        n, self.n, self.substeps = s.n_bodies, s.n_bodies, s.substeps
        self.joint_iterations = s.joint_iterations
        self.gravity = f(s.gravity)
        self.pos, self.pos_old, self.vel = f(s.pos), f(s.pos), torch.zeros(n, 2, dtype=torch.float64, device=dev)
        self.rot = f(s.rotation)
        self.vreq = f(s.vreq)
        self.static = i(s.body_type) == 1
        off = s.world_body_offsets if s.world_body_offsets is not None else np.array([0, n])
        self.world = torch.repeat_interleave(torch.arange(len(off) - 1, device=dev), i(np.diff(off.astype(np.int64))))
        self.box = f(s.world_box)[self.world]
        first = torch.full((len(off) - 1,), n, dtype=torch.int64, device=dev)
        dyn = torch.nonzero(~self.static).flatten()
        first.scatter_reduce_(0, self.world[dyn], dyn, "amin")
        self.first = first[first < n]
        self.parent, self.off, self.rad = i(s.col_parent), f(s.col_offset), f(s.col_radius)
        self.mass = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, self.parent, 4.0 * self.rad)
        reach = self.off.norm(dim=1) + self.rad
        self.bound = torch.zeros(n, dtype=torch.float64, device=dev).scatter_reduce_(0, self.parent, reach, "amax")
        self.spring = (i(s.spr_a), i(s.spr_b), f(s.spr_rest), f(s.spr_k), f(s.spr_c))
        # joints in arena order: those of a level touch different bodies
        last, level = {}, np.zeros(s.n_joints, np.int64)
        for j, (a, b) in enumerate(zip(s.jnt_a.tolist(), s.jnt_b.tolist())):
            level[j] = last[a] = last[b] = max(last.get(a, -1), last.get(b, -1)) + 1
        self.levels = [i(np.flatnonzero(level == k)) for k in range(int(level.max()) + 1)] if s.n_joints else []
        self.joint = (i(s.jnt_a), i(s.jnt_b), f(s.jnt_anchor_a), f(s.jnt_anchor_b), f(s.jnt_distance), f(s.jnt_target))
        self.snap = self._snapshots()
        self.old_dt, self.pending = 1.0, True

    def _snapshots(self):
        c, s = torch.cos(self.rot)[self.parent], torch.sin(self.rot)[self.parent]
        o = self.off
        return torch.stack([c * o[:, 0] - s * o[:, 1], s * o[:, 0] + c * o[:, 1]], 1) + self.pos[self.parent]

    @torch.no_grad()
    def _contacts(self):
        """Collider pairs (hi, lo) of different bodies that touch."""
        p, dev = self.snap, self.dev
        cell = torch.floor((p - p.min(0).values) / (2.0 * self.rad.max() * 1.0001)).long() + 1
        width, height = (cell.max(0).values + 3).tolist()
        key = ((self.world[self.parent] * height) + cell[:, 1]) * width + cell[:, 0]
        key, order = torch.sort(key)
        at = torch.arange(len(key), device=dev)
        hi, lo = [], []
        for step in (0, 1, width - 1, width, width + 1):
            b = at + 1 if step == 0 else torch.searchsorted(key, key + step)
            e = torch.searchsorted(key, key + step, right=True)
            m = (e - b).clamp(min=0)
            i = torch.repeat_interleave(at, m)
            j = torch.arange(len(i), device=dev) - torch.repeat_interleave(torch.cumsum(m, 0) - m, m) + b[i]
            i, j = order[i], order[j]
            d = (p[i] - p[j]).norm(dim=1)
            ok = (d < self.rad[i] + self.rad[j]) & (self.parent[i] != self.parent[j])
            hi.append(torch.maximum(i[ok], j[ok]))
            lo.append(torch.minimum(i[ok], j[ok]))
        return torch.cat(hi), torch.cat(lo)

    def substep(self, dt):
        p, m = self.pos, self.mass
        acc = self.gravity.expand(self.n, 2)
        a, b, rest, k, c = self.spring
        if len(a):
            d = p[b] - p[a]
            dist = d.norm(dim=1, keepdim=True)
            e = d / dist
            damp = e * (c[:, None] * ((self.vel[a] - self.vel[b]) * e).sum(1, keepdim=True))
            f = e * (k[:, None] * (dist - rest[:, None]) - damp)
            acc = acc.index_add(0, a, f / m[a][:, None]).index_add(0, b, -f / m[b][:, None])
        hi, lo = self._contacts()
        axis = self.snap[hi] - self.snap[lo]
        d = axis.norm(dim=1, keepdim=True)
        ph, pl = self.parent[hi], self.parent[lo]
        ratio = 1.0 - (m[ph] / (m[ph] + m[pl]))[:, None]
        push = axis / d * ((self.rad[hi] + self.rad[lo])[:, None] - d)
        p = p.index_add(0, ph, push * ratio).index_add(0, pl, -push * (1.0 - ratio))
        rot = self.rot
        a, b, aa, ab, dist, target = self.joint
        for _ in range(self.joint_iterations if self.levels else 0):
            for q in self.levels:
                ja, jb = a[q], b[q]
                dp = (p[jb] + ab[q]) - (p[ja] + aa[q])
                d = dp.norm(dim=1, keepdim=True)
                corr = (d - dist[q][:, None]) * dp / d
                ia, ib = 1.0 / m[ja], 1.0 / m[jb]
                share = (ia / (ia + ib))[:, None]
                p = p.index_add(0, ja, corr * share).index_add(0, jb, -corr * (1.0 - share))
                rc = 0.5 * (-torch.atan2(dp[:, 1], -dp[:, 0]) - torch.atan2(dp[:, 1], dp[:, 0]) - target[q])
                rot = rot.index_add(0, ja, rc * dt).index_add(0, jb, -rc * dt)
        self.rot = rot
        po = self.pos_old
        if self.pending:
            po = p - self.vreq * dt
        ratio = torch.ones(self.n, 1, dtype=torch.float64, device=self.dev)
        ratio[self.first] = dt / self.old_dt
        disp = (p - po) * ratio
        still = self.static[:, None]
        new = torch.where(still, p, p + disp + acc * dt * dt)
        self.vel = torch.where(still, torch.zeros_like(disp), disp / dt)
        self.pos_old, self.pos = p, new
        self.snap = self._snapshots()
        lo, hi = self.box[:, :2] + self.bound[:, None], self.box[:, 2:] - self.bound[:, None]
        self.pos = torch.minimum(torch.maximum(new, lo), hi)
        self.old_dt, self.pending = dt, False

    def step(self, dt):
        for _ in range(self.substeps):
            self.substep(float(np.float32(dt)) / self.substeps)


def exact(case, seed):
    kind = case["kind"]
    if kind == "hash":
        return None  # whole numbers
    s = _scene(case, seed)
    if kind == "gradient":
        if case["steps"] > 2 or case["worlds"] * case["n"] > 20_000:
            return None  # past the horizon over which the trajectories agree, or of what a tape of it can hold
        x = _Exact(s)
        x.vreq.requires_grad_()
        x.spring[3].requires_grad_()
        marked, target = _targets(case, seed, s)
        for _ in range(case["steps"]):
            x.step(s.dt)
        d = x.pos[torch.from_numpy(marked).to(x.dev)] - torch.from_numpy(target.astype(np.float64)).to(x.dev)
        dv, dk = torch.autograd.grad((d * d).sum() / len(marked), (x.vreq, x.spring[3]))
        return {"pos": x.pos.detach(), "dv": dv, "dk": dk}
    crowd = case.get("packing", 0.0) + case.get("springs", 0.0)
    if case["steps"] > 4 or crowd > 0.6 or (case["steps"] > 1 and crowd > 0.4):
        return None  # pushed apart from deep overlaps, or pulled together: the trajectories part at once
    with torch.no_grad():
        x = _Exact(s)
        for _ in range(1 + case["steps"]):
            x.step(s.dt)
    out = {"pos": x.pos, "pos_old": x.pos_old, "vel": x.vel if case["steps"] == 1 and crowd < 0.2 else None}
    if kind == "events":  # whole numbers; a pair at its threshold is in one trajectory's list and not in the other's
        out.update(n_events=None, a=None, b=None, va=None, vb=None)
    if kind == "jointed":
        out["rotation"] = x.rot
    return out
