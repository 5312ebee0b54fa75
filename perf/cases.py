"""Performance cases: the work that users of the library have it do, through its Python interface.

The sizes are those of the repository's workloads (serving stream: Plummer clusters of 256 to 65,536
bodies, direct sum up to 8,192; two Plummer spheres of 1,048,576 bodies at theta 0.5; the uniform cube
of 4,194,304 bodies with cell = cutoff = 2) and odd sizes between them.  All inputs come from the seed.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "nbody-gpu-sim_gb300"))

import nbgb  # noqa: E402
from nbgb.serving import Ensemble  # noqa: E402

EPS = 0.01


def listed():
    return [
        # A small simulation advanced a few steps between snapshots: launches and latency.
        {"name": "steps_direct_1k", "kind": "steps_direct", "n": 1024, "steps": 10},
        # Drop-in direct forces of a small system of odd size.
        {"name": "forces_direct_3k", "kind": "direct", "n": 3001, "compensated": True},
        # Drop-in direct forces of a large system: arithmetic.
        {"name": "forces_direct_131k", "kind": "direct", "n": 131072, "compensated": True},
        # The drop-in Barnes-Hut calculator (reference walk) on a medium system of odd size.
        {"name": "forces_bh_20k", "kind": "bh", "n": 20011, "walk": "reference", "leaf": 1,
         "theta": 0.5, "two": False},
        # The same on the large Barnes-Hut workload.
        {"name": "forces_bh_1m", "kind": "bh", "n": 1048576, "walk": "reference", "leaf": 1,
         "theta": 0.5, "two": True},
        # The group walk on the large Barnes-Hut workload.
        {"name": "forces_bh_group_1m", "kind": "bh", "n": 1048576, "walk": "group", "leaf": 1,
         "theta": 0.5, "two": True},
        # The group walk with 8-body buckets between those sizes.
        {"name": "forces_bh_group8_200k", "kind": "bh", "n": 200003, "walk": "group", "leaf": 8,
         "theta": 0.5, "two": True},
        # A serving-size Barnes-Hut simulation advanced a few steps between snapshots.
        {"name": "steps_bh_50k", "kind": "steps_bh", "n": 50021, "steps": 5},
        # The spatial hash on the uniform cube.
        {"name": "forces_hash_4m", "kind": "hash", "n": 4194304},
        # The drop-in FP32 integrator over the spatial hash, in the reference's ball of radius 10.
        {"name": "integrate_hash_60k", "kind": "integrate_hash", "n": 60013},
        # The energy monitor of a small simulation (FP64).
        {"name": "energy_8k", "kind": "energy", "n": 8191},
        # A burst of requests served from submission to the last result.
        {"name": "serve_burst_24", "kind": "serve", "systems": 24, "steps": 20},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["steps_direct", "direct", "bh", "bh", "steps_bh", "hash", "integrate_hash",
                       "energy", "serve"])
    if kind == "steps_direct":
        return {"kind": kind, "n": size(256, 8192), "steps": rng.randint(4, 20)}
    if kind == "direct":
        return {"kind": kind, "n": size(500, 131072), "compensated": rng.random() < 0.75}
    if kind == "bh":
        return {"kind": kind, "n": size(3000, 1000000), "walk": rng.choice(["reference", "group"]),
                "leaf": rng.choice([1, 1, 8]), "theta": rng.choice([0.5, 0.5, 0.75]),
                "two": rng.random() < 0.5}
    if kind == "steps_bh":
        return {"kind": kind, "n": size(8193, 65536), "steps": rng.randint(2, 8)}
    if kind == "hash":
        return {"kind": kind, "n": size(5000, 4000000)}
    if kind == "integrate_hash":
        return {"kind": kind, "n": size(2000, 100000)}
    if kind == "energy":
        return {"kind": kind, "n": size(256, 16384)}
    return {"kind": "serve", "systems": rng.randint(6, 24), "steps": rng.randint(10, 20)}


# ------------------------------------------------------------------ inputs --
def _generator(seed, *more):
    s = int(seed)
    for m in more:
        s = s * 1000003 + int(m)
    g = torch.Generator(device="cuda")
    g.manual_seed(s % (1 << 62))
    return g


def _isotropic(g, n):
    u = torch.rand((2, n), generator=g, device="cuda", dtype=torch.float64)
    c = 2.0 * u[0] - 1.0
    s = torch.sqrt(torch.clamp(1.0 - c * c, min=0.0))
    phi = 2.0 * math.pi * u[1]
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), c])


def _plummer(g, n, mass=1.0):
    """Positions and velocities (3, n) of an equal-mass Plummer sphere (a = 1, G = 1)."""
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64).clamp_(1e-12, 1.0 - 1e-12)
    r = 1.0 / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
    q = torch.linspace(0.0, 1.0, 4097, device="cuda", dtype=torch.float64)
    f = q * q * (1.0 - q * q) ** 3.5
    cdf = torch.cat([f.new_zeros(1), torch.cumsum(0.5 * (f[1:] + f[:-1]), 0)])
    cdf = cdf / cdf[-1].clone()
    t = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    k = torch.searchsorted(cdf, t).clamp_(1, 4096)
    w = (t - cdf[k - 1]) / (cdf[k] - cdf[k - 1]).clamp(min=1e-300)
    speed = (q[k - 1] + w * (q[k] - q[k - 1])) * math.sqrt(2.0 * mass) * (r * r + 1.0) ** -0.25
    return _isotropic(g, n) * r, _isotropic(g, n) * speed


def _bodies(case, seed):
    """x, y, z, vx, vy, vz, m as float32 tensors on the GPU."""
    n, kind = case["n"], case["kind"]
    g = _generator(seed, n)
    mass = torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)
    if kind == "hash":  # uniform cube at the workload's density
        side = 160.0 * (n / 4194304.0) ** (1.0 / 3.0)
        x = torch.rand((3, n), generator=g, device="cuda", dtype=torch.float64) * side
        v = torch.zeros_like(x)
    elif kind == "integrate_hash":  # uniform ball of radius 10
        u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
        x = _isotropic(g, n) * (10.0 * u ** (1.0 / 3.0))
        v = 0.05 * torch.randn((3, n), generator=g, device="cuda", dtype=torch.float64)
        mass = mass * (0.5 + torch.rand(n, generator=g, device="cuda", dtype=torch.float64))
    elif case.get("two"):  # two spheres of half the mass, 10 apart, approaching
        h = n // 2
        xa, va = _plummer(g, h, 0.5)
        xb, vb = _plummer(g, n - h, 0.5)
        xa[0] -= 5.0
        xb[0] += 5.0
        va[0] += 0.15
        vb[0] -= 0.15
        x, v = torch.cat([xa, xb], 1), torch.cat([va, vb], 1)
    else:
        x, v = _plummer(g, n)
    return [t.float().contiguous() for t in (x[0], x[1], x[2], v[0], v[1], v[2], mass)]


def _host_state(b):
    return {k: t.cpu().numpy() for k, t in zip(("x", "y", "z", "vx", "vy", "vz", "m"), b)}


def _device_view(fields, n):
    """A ParticleData over the caller's device tensors."""
    pd = nbgb.ParticleData(n)
    for name, t in fields.items():
        setattr(pd.struct, name, t.data_ptr())
    pd.on_device = True
    return pd


def _requests(case, seed):
    """The serving stream's systems: N log-uniform in [256, 65536]."""
    rng = np.random.Generator(np.random.PCG64(1000 + case["systems"]))
    ns = np.exp(rng.uniform(math.log(256), math.log(65536), case["systems"])).round().astype(int)
    return [_bodies({"kind": "serve", "n": int(n)}, seed * 64 + i) for i, n in enumerate(ns)]


SERVE_DT = 1e-4
STEP_DT = 1e-4
HASH_DT = 1e-3


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "serve":
        s["requests"] = [_host_state(b) for b in _requests(case, seed)]
        s["ensemble"] = Ensemble(hbm_budget_bytes=4 << 30, softening=EPS, theta=0.5)
        return s
    n = case["n"]
    b = _bodies(case, seed)
    if kind in ("steps_direct", "energy", "steps_bh"):
        if kind == "steps_bh":
            calc = nbgb.BarnesHutCalculator(0.5, group_walk=True)
            calc.set_flags(calc.params.flags & ~nbgb.FLAG_SYNC)
        else:
            calc = nbgb.DirectForceCalculator()
        calc.setSofteningParameter(EPS)
        s["calc"] = calc
        s["system"] = nbgb.System(calc, _host_state(b))
        return s
    f = dict(zip(("pos_x", "pos_y", "pos_z", "vel_x", "vel_y", "vel_z", "mass"), b))
    for k in ("acc_x", "acc_y", "acc_z", "acc_old_x", "acc_old_y", "acc_old_z"):
        f[k] = torch.zeros(n, device="cuda")
    if kind == "direct":
        calc = nbgb.DirectForceCalculator()
        if not case["compensated"]:
            calc.set_flags(calc.params.flags & ~nbgb.FLAG_COMPENSATED)
    elif kind == "bh":
        calc = nbgb.BarnesHutCalculator(case["theta"], leaf_capacity=case["leaf"],
                                        group_walk=case["walk"] == "group")
    else:
        calc = nbgb.SpatialHashCalculator(2.0, 2.0)
    calc.setSofteningParameter(EPS)
    s.update(calc=calc, fields=f, particles=_device_view(f, n))
    torch.cuda.current_stream().synchronize()
    if kind == "integrate_hash":  # a(0), as after the first frame
        s["integrator"] = nbgb.Integrator()
        calc.computeForces(s["particles"])
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("direct", "bh", "hash"):
        state["calc"].computeForces(state["particles"])
        return [state["fields"][k] for k in ("acc_x", "acc_y", "acc_z")]
    if kind == "integrate_hash":
        state["integrator"].integrate(state["particles"], state["calc"], HASH_DT)
        return [state["fields"][k] for k in ("pos_x", "pos_y", "pos_z", "vel_x", "vel_y", "vel_z",
                                             "acc_x", "acc_y", "acc_z")]
    if kind == "energy":
        ke, pe, mom = state["system"].energy()
        return [ke, pe, mom]
    if kind in ("steps_direct", "steps_bh"):
        state["system"].step(STEP_DT, case["steps"])
        return state["system"].read_f64()
    ens = state["ensemble"]
    ids = [ens.submit(r, case["steps"], SERVE_DT) for r in state["requests"]]
    done = {}
    while ens.tick() != (0, 0):
        while (got := ens.poll(want_state=True)) is not None:
            done[got[0]["request_id"]] = got[1]
    ens.synchronize()
    while (got := ens.poll(want_state=True)) is not None:
        done[got[0]["request_id"]] = got[1]
    return {k: np.concatenate([done[i][k] for i in ids]) for k in ("x", "y", "z", "vx", "vy", "vz")}


# -------------------------------------------------------------------- work --
def _interactions(n, theta=0.5):
    """Accepted interactions per body of the reference's opening rule (counted: 1,679 at 27 K,
    2,587 at 1 M bodies, theta 0.5)."""
    if n <= 1:
        return 0.0
    return min(n - 1.0, max(20.0, 171.0 * math.log2(n) - 833.0) * (0.5 / theta) ** 2)


def work(case):
    """20 flops per interaction (the pair law), 30 per FP64 pair of the energy; bodies in, results out."""
    kind = case["kind"]
    if kind == "serve":
        rng = np.random.Generator(np.random.PCG64(1000 + case["systems"]))
        ns = np.exp(rng.uniform(math.log(256), math.log(65536), case["systems"])).round()
        it = sum(n * ((n - 1) if n <= 8192 else _interactions(n)) for n in ns)
        return {"bytes": float(ns.sum()) * (28 + 48 + 124 * (case["steps"] + 1)),
                "flops": 20.0 * it * (case["steps"] + 1)}
    n = float(case["n"])
    if kind == "steps_direct":
        return {"bytes": n * (124 * case["steps"] + 48), "flops": 20.0 * n * (n - 1) * case["steps"]}
    if kind == "steps_bh":
        return {"bytes": n * (124 * case["steps"] + 48),
                "flops": 20.0 * n * _interactions(n) * case["steps"]}
    if kind == "direct":
        return {"bytes": 28.0 * n, "flops": 20.0 * n * (n - 1)}
    if kind == "bh":
        return {"bytes": 28.0 * n, "flops": 20.0 * n * _interactions(n, case["theta"])}
    if kind == "hash":  # about 34 neighbours within the cutoff of 221 candidates
        return {"bytes": 28.0 * n, "flops": n * (221 * 8 + 34 * 12.0)}
    if kind == "integrate_hash":  # candidates: 27 cells of 8 in a ball of volume 4189
        cand = 27 * 8 * n / 4189.0
        return {"bytes": 124.0 * n, "flops": n * cand * (8 + 0.155 * 12)}
    return {"bytes": 64.0 * n, "flops": 15.0 * n * (n - 1)}


# ------------------------------------------------------------------- exact --
def _direct64(x, y, z, m, eps):
    """FP64 direct sum over all bodies (float64 tensors)."""
    n = x.numel()
    out = torch.empty((3, n), device="cuda", dtype=torch.float64)
    rows = max(1, min(n, (1 << 27) // max(n, 1)))
    for a in range(0, n, rows):
        b = min(n, a + rows)
        dx, dy, dz = x[None] - x[a:b, None], y[None] - y[a:b, None], z[None] - z[a:b, None]
        f = dx * dx
        f.addcmul_(dy, dy).addcmul_(dz, dz).add_(eps * eps)
        f = torch.rsqrt(f).pow_(3).mul_(m[None])
        out[0, a:b] = (f * dx).sum(1)
        out[1, a:b] = (f * dy).sum(1)
        out[2, a:b] = (f * dz).sum(1)
    return out


def _kdk64(b, dt, steps, eps):
    """Kick-drift-kick in FP64 from the FP32 initial state; the state after `steps` steps."""
    x, y, z, vx, vy, vz, m = (t.double() for t in b)
    p, v = torch.stack([x, y, z]), torch.stack([vx, vy, vz])
    a = _direct64(p[0], p[1], p[2], m, eps)
    for _ in range(steps):
        v = v + 0.5 * dt * a
        p = p + dt * v
        a = _direct64(p[0], p[1], p[2], m, eps)
        v = v + 0.5 * dt * a
    return dict(zip(("x", "y", "z", "vx", "vy", "vz"), (*p, *v)))


def _cutoff64(x, y, z, m, cutoff, eps):
    """Forces within the cutoff: neighbours by the law's float32 test d^2 < cutoff^2 (d^2 = fma(dz, dz,
    fma(dy, dy, dx dx))), sums in FP64."""
    p = torch.stack([x, y, z])
    lo = p.double().amin(1) - 0.001
    cell = 1.001 * cutoff
    c = torch.floor((p.double() - lo[:, None]) / cell).long()
    d = [int(v) + 1 for v in c.amax(1).tolist()]
    key = c[0] + d[0] * (c[1] + d[1] * c[2])
    order = torch.argsort(key, stable=True)
    key, p, w, c = key[order], p[:, order], m[order].double(), c[:, order]
    start = torch.searchsorted(key, torch.arange(d[0] * d[1] * d[2] + 1, device="cuda"))
    n = x.numel()
    me = torch.arange(n, device="cuda")
    cut2 = float(np.float32(cutoff) * np.float32(cutoff))
    acc = torch.zeros((3, n), device="cuda", dtype=torch.float64)
    for oz in (-1, 0, 1):
        for oy in (-1, 0, 1):
            cy, cz = c[1] + oy, c[2] + oz
            ok = (cy >= 0) & (cy < d[1]) & (cz >= 0) & (cz < d[2])
            row = d[0] * (cy.clamp(0, d[1] - 1) + d[1] * cz.clamp(0, d[2] - 1))
            s = start[row + (c[0] - 1).clamp(min=0)]
            e = torch.where(ok, start[row + (c[0] + 1).clamp(max=d[0] - 1) + 1], s)
            for t in range(int((e - s).max())):
                j = (s + t).clamp(max=n - 1)
                dx, dy, dz = p[0, j] - p[0], p[1, j] - p[1], p[2, j] - p[2]
                t1 = (dx.double() ** 2).float()
                t2 = (dy.double() ** 2 + t1.double()).float()
                d2 = (dz.double() ** 2 + t2.double()).float()
                use = (s + t < e) & (d2 < cut2) & (j != me)
                q = p[:, j].double() - p.double()
                f = torch.where(use, w[j] * ((q * q).sum(0) + eps * eps) ** -1.5, 0.0)
                acc += f * q
    out = torch.empty_like(acc)
    out[:, order] = acc
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        got = [_kdk64(b, float(np.float32(SERVE_DT)), case["steps"], float(np.float32(EPS)))
               for b in _requests(case, seed)]
        return {k: torch.cat([g[k] for g in got]) for k in ("x", "y", "z", "vx", "vy", "vz")}
    eps = float(np.float32(EPS))
    b = _bodies(case, seed)
    if kind in ("steps_direct", "steps_bh"):
        return _kdk64(b, float(np.float32(STEP_DT)), case["steps"], eps)
    if kind in ("direct", "bh"):
        if case["n"] > 400000:
            return None
        return list(_direct64(*(b[k].double() for k in (0, 1, 2, 6)), eps))
    if kind == "hash":
        return list(_cutoff64(b[0], b[1], b[2], b[6], 2.0, eps))
    if kind == "integrate_hash":
        dt = np.float32(HASH_DT)
        half = float(np.float32(0.5) * dt * dt)
        a0 = _cutoff64(b[0], b[1], b[2], b[6], 2.0, eps).float()
        pos = []
        for k in range(3):  # the float32 position update, whose result the forces see
            t = (a0[k].double() * half).float()
            pos.append(b[k] + (b[3 + k].double() * float(dt) + t.double()).float())
        a1 = _cutoff64(*pos, b[6], 2.0, eps)
        vel = [b[3 + k].double() + 0.5 * float(dt) * (a0[k].double() + a1[k]) for k in range(3)]
        return [*(t.double() for t in pos), *vel, *a1]
    x, y, z, vx, vy, vz, m = (t.double() for t in b)
    ke = float((0.5 * m * (vx * vx + vy * vy + vz * vz)).sum())
    pe = 0.0
    n = case["n"]
    for a in range(0, n, 1024):
        q = slice(a, min(n, a + 1024))
        r2 = (x[None] - x[q, None]) ** 2 + (y[None] - y[q, None]) ** 2 + (z[None] - z[q, None]) ** 2
        phi = (m[None] * torch.rsqrt(r2 + eps * eps)).sum(1) - m[q] / eps
        pe -= 0.5 * float((m[q] * phi).sum())
    mom = np.array([float((m * v).sum()) for v in (vx, vy, vz)])
    return [ke, pe, mom]
