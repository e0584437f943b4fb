"""Work that users of the library have it do, as timed cases.

Every case goes through the public entry points: a handle stepped in device
memory (`Simulation.step`, `nb_get_device_view`), a rendered frame
(`Simulation.update`, `copy_vertices`), steps followed by a snapshot in host
memory (`Simulation.positions`), a batch (`Batch.step`, `Batch.get_state`), a
burst of served jobs (`Server.submit`, `wait`, `result`) and the allocation-free
accelerations (`nb_direct_accel_noalloc`).  A pass advances its state, as a
simulation does; the same state can be run again.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import nbodysimulation_gb300 as nb

ALGO = {"tree": nb.BARNES_HUT, "global": nb.BRUTE_FORCE_GLOBAL, "tiled": nb.BRUTE_FORCE_LOCAL}
METHOD = {"euler": nb.EULER, "kdk": nb.KDK_LEAPFROG}
N_MAX = 4194304
DIRECT_BELOW = 8192  # batched and served systems below this size take the direct sum


def listed():
    return [
        # the smallest call: accelerations for a host engine's few hundred
        # bodies, once per frame, odd count; latency is all there is
        {"name": "accel_777", "kind": "accel", "n": 777, "eps": 0.01},
        # the plain direct sum at the size the reference runs it, 20 steps a call
        {"name": "direct_global_4096", "kind": "steps", "algo": "global", "n": 4096, "dist": "normal", "eps": 0.05,
         "theta": 0.5, "method": "euler", "multipole": 0, "precision": 0, "collision": False, "steps": 20,
         "read": "device"},
        # one rendered frame of the reference's default configuration:
        # 20,000 bodies, its masses and G, frame-time rule, vertices read back
        {"name": "frame_20000", "kind": "frame", "n": 20000, "algo": "global"},
        # a middle-sized direct sum with an odd count, leapfrog
        {"name": "direct_tiled_50021", "kind": "steps", "algo": "tiled", "n": 50021, "dist": "normal", "eps": 0.01,
         "theta": 0.5, "method": "kdk", "multipole": 0, "precision": 0, "collision": False, "steps": 1,
         "read": "device"},
        # the largest direct sum: exact forces of a system the tree also runs
        {"name": "direct_tiled_262144", "kind": "steps", "algo": "tiled", "n": 262144, "dist": "ball", "eps": 0.01,
         "theta": 0.5, "method": "euler", "multipole": 0, "precision": 0, "collision": False, "steps": 1,
         "read": "device"},
        # a small tree, odd count: every stage is short, launches and latency count
        {"name": "tree_6007", "kind": "steps", "algo": "tree", "n": 6007, "dist": "ball", "eps": 0.01, "theta": 0.5,
         "method": "euler", "multipole": 0, "precision": 0, "collision": False, "steps": 10, "read": "device"},
        # the plain Barnes-Hut configuration: unit ball in rotation, monopoles, FP32 sums
        {"name": "tree_ball_262144", "kind": "steps", "algo": "tree", "n": 262144, "dist": "ball", "eps": 0.01,
         "theta": 0.5, "method": "euler", "multipole": 0, "precision": 0, "collision": False, "steps": 1,
         "read": "device"},
        # a production run: leapfrog, quadrupoles, odd count, a snapshot in host memory every 4 steps
        {"name": "tree_kdk_100003", "kind": "steps", "algo": "tree", "n": 100003, "dist": "normal", "eps": 0.01,
         "theta": 0.7, "method": "kdk", "multipole": 1, "precision": 0, "collision": False, "steps": 4,
         "read": "host"},
        # the precision configuration, the largest: 4M bodies of a flat
        # system, lognormal masses, quadrupoles, compensated sums
        {"name": "tree_flat_4194304", "kind": "steps", "algo": "tree", "n": N_MAX, "dist": "flat", "eps": 0.005,
         "theta": 0.5, "method": "euler", "multipole": 1, "precision": 1, "collision": False, "steps": 1,
         "read": "device"},
        # the collision update after the tree step, as the reference's option runs it
        {"name": "collide_131072", "kind": "steps", "algo": "tree", "n": 131072, "dist": "ball", "eps": 0.01,
         "theta": 0.5, "method": "euler", "multipole": 0, "precision": 0, "collision": True, "steps": 1,
         "read": "device"},
        # many independent systems of uneven size in one batch, states read at the end
        {"name": "batch_48", "kind": "batch", "systems": 48, "n_max": 32768, "steps": 4, "theta": 0.5},
        # a burst of jobs through the job server, final states fetched
        {"name": "serve_10", "kind": "serve", "jobs": 10, "n_max": 32768, "steps_max": 30},
    ]


def _size(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, n | 1 if rng.random() < 0.6 else n))


def draw(rng):
    kind = rng.choice(["accel", "frame", "direct", "direct", "tree", "tree", "tree", "collide", "batch", "serve"])
    if kind == "accel":
        return {"kind": "accel", "n": _size(rng, 256, nb.NOALLOC_MAX_BODIES), "eps": rng.choice([0.0, 0.01, 0.05])}
    if kind == "frame":
        return {"kind": "frame", "n": _size(rng, 1000, 60000), "algo": rng.choice(["global", "tiled", "tree"])}
    if kind == "batch":
        return {"kind": "batch", "systems": rng.randint(6, 48), "n_max": _size(rng, 4096, 32768),
                "steps": rng.randint(1, 4), "theta": rng.choice([0.5, 0.7])}
    if kind == "serve":
        return {"kind": "serve", "jobs": rng.randint(3, 10), "n_max": _size(rng, 4096, 32768),
                "steps_max": rng.randint(12, 30)}
    case = {"kind": "steps", "algo": "tree", "dist": rng.choice(["ball", "normal", "flat"]),
            "eps": rng.choice([0.005, 0.01, 0.05]), "theta": rng.choice([0.5, 0.7, 0.8]),
            "method": rng.choice(["euler", "kdk"]), "multipole": rng.randint(0, 1), "precision": rng.randint(0, 1),
            "collision": False, "read": rng.choice(["device", "host"])}
    if kind == "direct":
        case["n"] = _size(rng, 1024, 200000)
        case |= {"algo": rng.choice(["global", "tiled"]), "multipole": 0, "precision": 0,
                 "steps": rng.randint(1, 10) if case["n"] < 40000 else 1}
    elif kind == "collide":
        case["n"] = _size(rng, 2000, 131072)
        case |= {"collision": True, "dist": "ball", "steps": 1, "algo": rng.choice(["tree", "tiled"])}
    else:
        case["n"] = _size(rng, 1024, 2000000)
        case["steps"] = rng.randint(1, 10) if case["n"] < 300000 else 1
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _bodies(dist, n, seed):
    """(pos[n,3], vel[n,3], mass[n]) float32 tensors."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(0x9E3779B1 * (seed + 1) % (1 << 62) + n)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=dev, dtype=torch.float32)

    mass = torch.full((n,), 1.0 / n, dtype=torch.float32, device=dev)
    if dist == "ball":  # uniform in the unit ball, rotating about z with the enclosed mass r^3
        d = normal(n, 3)
        r = torch.rand(n, 1, generator=g, device=dev, dtype=torch.float32).pow(1.0 / 3.0)
        pos = d / d.norm(dim=1, keepdim=True).clamp_min(1e-20) * r
        rho = pos[:, :2].norm(dim=1, keepdim=True).clamp_min(1e-20)
        vel = torch.cat([-pos[:, 1:2], pos[:, 0:1], torch.zeros_like(rho)], 1) / rho * r
    elif dist == "flat":  # flat normal system, lognormal masses
        pos = normal(n, 3) * torch.tensor([1.0, 1.0, 0.2], device=dev)
        vel = torch.zeros_like(pos)
        m = torch.exp(0.5 * normal(n).double())
        mass = (m / m.sum()).float()
    elif dist == "reference":  # the reference's defaults: normal(0, 1.5), |normal(0.5, 0.25)| masses
        pos = normal(n, 3) * 1.5
        vel = torch.zeros_like(pos)
        mass = (0.5 + 0.25 * normal(n)).abs()
    else:
        pos = normal(n, 3)
        vel = torch.zeros_like(pos)
    return pos.contiguous(), vel.contiguous(), mass.contiguous()


def _systems(case, seed):
    """[(n, dist, seed, steps)] of a batch or a burst: sizes log-uniform from
    1024 to n_max, half normal, half ball."""
    r = np.random.default_rng(1000003 * seed + 17)
    many = case["systems"] if case["kind"] == "batch" else case["jobs"]
    # the same sizes for every seed, so that a pass is the same work
    s = np.random.default_rng(29 * many + case["n_max"])
    n = np.exp(s.uniform(math.log(1024), math.log(case["n_max"]), many)).astype(int)
    n[0] = case["n_max"]
    steps = s.integers(10, case["steps_max"] + 1, many) if case["kind"] == "serve" else [case["steps"]] * many
    return [(int(n[k]), "ball" if k % 2 else "normal", int(r.integers(1 << 30)), int(steps[k])) for k in range(many)]


def _system_config(n, theta):
    return nb.default_config(num_of_bodies=n, gravitational_constant=1.0, theta=theta, epsilon=0.01,
                             algo_config=nb.BRUTE_FORCE_LOCAL if n < DIRECT_BELOW else nb.BARNES_HUT,
                             numerical_method=nb.EULER)


DT = 1e-3
FRAME_DT = 1.0 / 60.0  # clamped to 0.005 by the frame-time rule
JOB_THETA = 0.5


class _DeviceArray:
    """float32[n, 4] of device memory that `owner` holds, for torch.as_tensor."""

    def __init__(self, ptr, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n, 4), "typestr": "<f4", "data": (ptr, False), "version": 3}


class _Views:
    """Tensors over a handle's device arrays, made once per array."""

    def __init__(self, sim):
        self.sim, self.made = sim, {}

    def get(self, ptr):
        if ptr not in self.made:
            self.made[ptr] = torch.as_tensor(_DeviceArray(ptr, self.sim.n, self.sim), device="cuda")
        return self.made[ptr]

    def state(self):
        v = self.sim.device_view()
        return self.get(v.body_pm), self.get(v.vel), self.get(v.acc)


def _set_device_state(sim, pos, vel, mass):
    torch.cuda.synchronize()
    st = sim.L.nb_set_state_device(sim.h, pos.data_ptr(), vel.data_ptr(), mass.data_ptr())
    if st:
        raise nb.NbError(st, "nb_set_state_device")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "accel":
        pos, _, mass = _bodies("normal", case["n"], seed)
        body = torch.cat([pos, mass[:, None]], 1).contiguous()
        return {"case": case, "L": nb.load(), "body": body, "acc": torch.empty_like(body)}
    if kind == "frame":
        sim = nb.Simulation(num_of_bodies=case["n"], algo_config=ALGO[case["algo"]])
        _set_device_state(sim, *_bodies("reference", case["n"], seed))
        return {"case": case, "sim": sim, "views": _Views(sim)}
    if kind == "steps":
        sim = nb.Simulation(num_of_bodies=case["n"], algo_config=ALGO[case["algo"]], theta=case["theta"],
                            epsilon=case["eps"], gravitational_constant=1.0,
                            numerical_method=METHOD[case["method"]], multipole=case["multipole"],
                            precision=case["precision"], collision=int(case["collision"]))
        _set_device_state(sim, *_bodies(case["dist"], case["n"], seed))
        host = tuple(np.zeros((case["n"], 3), np.float32) for _ in range(2)) if case["read"] == "host" else None
        return {"case": case, "sim": sim, "views": _Views(sim), "host": host}
    systems = _systems(case, seed)
    states = [[t.cpu().numpy() for t in _bodies(dist, n, s)] for n, dist, s, _ in systems]
    if kind == "batch":
        batch = nb.Batch([_system_config(n, case["theta"]) for n, *_ in systems])
        for k, (pos, vel, mass) in enumerate(states):
            batch.set_state(k, pos, mass, vel)
        total = sum(n for n, *_ in systems)
        out = [np.zeros((total, 3), np.float32) for _ in range(3)] + [np.zeros(total, np.float32)]
        return {"case": case, "batch": batch, "out": out}
    server = nb.Server(max_jobs=16, snapshot_every=0)
    return {"case": case, "server": server, "states": states,
            "jobs": [(_system_config(n, JOB_THETA), n, steps) for n, _, _, steps in systems]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "accel":
        st = state["L"].nb_direct_accel_noalloc(state["body"].data_ptr(), case["n"], case["eps"], 1.0,
                                                state["acc"].data_ptr(),
                                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st:
            raise nb.NbError(st, "nb_direct_accel_noalloc")
        return state["acc"]
    if kind == "frame":
        sim = state["sim"]
        sim.update(FRAME_DT)
        vertices = sim.copy_vertices()
        _, vel, acc = state["views"].state()
        return vertices, vel, acc
    if kind == "steps":
        sim = state["sim"]
        sim.step(DT, case["steps"])
        if state["host"] is not None:
            return sim.positions(with_velocities=True, out=state["host"])
        return state["views"].state()
    if kind == "batch":
        batch, out = state["batch"], state["out"]
        batch.step(DT, case["steps"])
        at = 0
        for k, n in enumerate(batch.ns):
            batch.get_state(k, out=tuple(a[at:at + n] for a in out))
            at += n
        return tuple(out)
    server = state["server"]
    ids = [server.submit(cfg, steps, DT, pos, mass, vel)
           for (cfg, _, steps), (pos, vel, mass) in zip(state["jobs"], state["states"])]
    status = server.wait()
    if status:
        raise nb.NbError(status, "nb_server_wait")
    return [server.result(job, n) for job, (_, n, _) in zip(ids, state["jobs"])]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
PAIR_FLOPS = 19          # difference 3, d^2 + eps^2 6, rsqrt 1, m / d^3 3, sum 6
QUADRUPOLE_FLOPS = 48    # the same with the traceless quadrupole term
BYTES_IN, BYTES_OUT = 28, 36  # position, velocity, mass; position, velocity, acceleration


def _flops(algo, n, theta, multipole, steps):
    if algo != "tree":
        return float(n) * n * steps * PAIR_FLOPS
    # interactions per body grow with log N and with the cone of open cells
    per_body = min(float(n), 110.0 * math.log2(max(n, 2)) * (0.5 / theta) ** 2)
    return n * steps * per_body * (0.25 * PAIR_FLOPS + 0.75 * (QUADRUPOLE_FLOPS if multipole else PAIR_FLOPS))


def work(case):
    kind = case["kind"]
    if kind == "accel":
        return {"bytes": 32.0 * case["n"], "flops": _flops("tiled", case["n"], 0, 0, 1)}
    if kind == "frame":
        n = case["n"]
        return {"bytes": (BYTES_IN + BYTES_OUT + 16.0) * n, "flops": _flops(case["algo"], n, 1.5, 0, 1)}
    if kind == "steps":
        n = case["n"]
        return {"bytes": float(BYTES_IN + BYTES_OUT) * n,
                "flops": _flops(case["algo"], n, case["theta"], case["multipole"], case["steps"])}
    systems = _systems(case, 0)
    return {"bytes": float(BYTES_IN + BYTES_OUT) * sum(n for n, *_ in systems),
            "flops": sum(_flops("tiled" if n < DIRECT_BELOW else "tree", n, case.get("theta", JOB_THETA), 0, steps)
                         for n, _, _, steps in systems)}


# ---------------------------------------------------------------------------
# the same in 64 bits: direct sums, also of the systems that the tree
# approximates
# ---------------------------------------------------------------------------
MOST_PAIRS = 7.5e10


def _accel64(pos, mass, eps, G):
    n = pos.shape[0]
    acc = torch.empty_like(pos)
    rows = max(1, min(n, (1 << 26) // n))
    for i in range(0, n, rows):
        p = pos[i:i + rows]
        d = [pos[None, :, c] - p[:, None, c] for c in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps * eps
        f = torch.where(r2 > 0, mass[None, :] * r2.clamp_min(1e-300).pow(-1.5), torch.zeros_like(r2))
        for c in range(3):
            acc[i:i + rows, c] = G * (f * d[c]).sum(1)
    return acc


def _advance64(pos, vel, mass, eps, G, dt, method, steps):
    eps, G, dt = float(np.float32(eps)), float(np.float32(G)), float(np.float32(dt))
    pos, vel, mass = pos.double(), vel.double(), mass.double()
    acc = torch.zeros_like(pos)
    for k in range(steps):
        acc = _accel64(pos, mass, eps, G)
        vel = vel + acc * (dt * (0.5 if method == "kdk" and k == 0 else 1.0))
        pos = pos + vel * dt
    return pos, vel, acc


def _quad(x, last):
    return torch.cat([x, last.reshape(-1, 1).expand(x.shape[0], 1)], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        systems = _systems(case, seed)
        if sum(float(n) * n * steps for n, _, _, steps in systems) > MOST_PAIRS:
            return None
        theirs = []
        for n, dist, s, steps in systems:
            pos, vel, mass = _bodies(dist, n, s)
            theirs.append(_advance64(pos, vel, mass, 0.01, 1.0, DT, "euler", steps) + (mass.double(),))
        if kind == "serve":
            return [(p.cpu().numpy(), v.cpu().numpy()) for p, v, *_ in theirs]
        return tuple(torch.cat([t[k] for t in theirs]).cpu().numpy() for k in range(4))
    n = case["n"]
    if float(n) * n * case.get("steps", 1) > MOST_PAIRS:
        return None
    zero = torch.zeros(1, dtype=torch.float64, device=_device())
    if kind == "accel":
        pos, _, mass = _bodies("normal", n, seed)
        return _quad(_accel64(pos.double(), mass.double(), float(np.float32(case["eps"])), 1.0), zero)
    if kind == "frame":
        p, v, a = _advance64(*_bodies("reference", n, seed), 0.01, 6.67e-11, 0.005, "euler", 1)
        return _quad(p, zero + 1.0).cpu().numpy(), _quad(v, zero), _quad(a, zero)
    pos, vel, mass = _bodies(case["dist"], n, seed)
    p, v, a = _advance64(pos, vel, mass, case["eps"], 1.0, DT, case["method"], case["steps"])
    if case["collision"]:  # reflections depend on contacts that rounding decides: positions and accelerations only
        v = None
    if case["read"] == "host":
        return p.cpu().numpy(), None if v is None else v.cpu().numpy()
    return _quad(p, mass.double()), None if v is None else _quad(v, zero), _quad(a, zero)
