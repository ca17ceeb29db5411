"""What the speed of this framework is measured on.

A case is one call, or one short loop of calls, of a user's program through
the package's public entry points, on inputs such a program has in hand:

* ``step``: one update of a flock that lives in the caller's device arrays
  (``boids_step_noalloc``), queued on the caller's stream;
* ``flock``: a flock kept by a ``BoidSimulation`` handle: its state set from
  host memory, ``steps`` updates, the state (and with ``forces`` the rule
  forces) read back, as between two frames of a recorded run;
* ``sweep``: a batched ensemble of flocks of uneven size drawn, run and
  scored by its order statistics, as a parameter sweep does per batch;
* ``predict`` and ``train``: the sweep's surrogate network, screening points
  and being fitted to simulated ones.

Flocks use the two parameter sets of the tests and the benchmark
(settings/marun2019.ini and settings/test.ini) at those sets' densities.
``age`` updates have passed since the seeded placement when a case begins: a
flock starts uniform and gathers into crowded groups, and users run both.
"""
import ctypes
import math

import numpy as np
import torch

import boidssimulatormpi_gb300 as B
from boidssimulatormpi_gb300.workload import MARUN2019

# settings/test.ini: wider cones, longer sight, 1000 boids per unit volume
TEST_INI = dict(sep=(0.1, 0.9, 0.0001), ali=(0.1, 0.7, 0.1), coh=(0.1, 0.8, 0.1), vmax=0.003, vmin=0.001)
SETS = {"marun2019": (MARUN2019, 16384.0, "random_uniform"), "test": (TEST_INI, 1000.0, "test")}


def listed():
    return [
        # the reference's own test flock stepped inside a host application: latency is everything
        {"name": "step_n1000", "kind": "step", "set": "test", "n": 1000, "age": 0},
        # the reference's CPU configuration, gathered, stepped inside a host application
        {"name": "step_n16384_gathered", "kind": "step", "set": "marun2019", "n": 16384, "age": 300},
        # near the largest flock the allocation-free step takes, an odd size, still uniform
        {"name": "step_n262143", "kind": "step", "set": "marun2019", "n": 262143, "age": 10},
        # the reference's compare_mpi.sh run: 1000 boids over 100 updates
        {"name": "flock_n1000_t100", "kind": "flock", "set": "test", "n": 1000, "age": 0, "steps": 100,
         "forces": False, "pairs": False},
        # the reference's CPU configuration over its horizon of 100 updates, from the placement
        {"name": "flock_n16384_t100", "kind": "flock", "set": "marun2019", "n": 16384, "age": 0, "steps": 100,
         "forces": False, "pairs": False},
        # a gathered flock of an odd size recorded with its forces every 10th update
        {"name": "flock_n65537_gathered_t10", "kind": "flock", "set": "marun2019", "n": 65537, "age": 400,
         "steps": 10, "forces": True, "pairs": False},
        # the benchmark's flock, every update with its state set and read back
        {"name": "flock_n1048576_t1", "kind": "flock", "set": "marun2019", "n": 1 << 20, "age": 5, "steps": 1,
         "forces": False, "pairs": False},
        # the benchmark's flock once it has gathered, recorded every 10th update
        {"name": "flock_n1048576_gathered_t10", "kind": "flock", "set": "marun2019", "n": 1 << 20, "age": 400,
         "steps": 10, "forces": False, "pairs": False},
        # the all-pairs engine on its own kernels, the reference's boidsim configuration
        {"name": "pairs_n65536_t3", "kind": "flock", "set": "marun2019", "n": 65536, "age": 30, "steps": 3,
         "forces": False, "pairs": True},
        # a batch of a parameter sweep
        {"name": "sweep_f48_t200", "kind": "sweep", "flocks": 48, "low": 1024, "high": 16384, "steps": 200},
        # a sweep's points screened by the surrogate
        {"name": "predict_r65536", "kind": "predict", "rows": 65536},
        # the surrogate fitted to a sweep's training runs
        {"name": "train_r1024_e30", "kind": "train", "rows": 1024, "epochs": 30, "batch": 256},
    ]


def _log(rng, low, high):
    """A whole number in [low, high], even over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(("step", "step", "flock", "flock", "flock", "pairs", "sweep", "predict", "train"))
    if kind == "step":
        if rng.random() < 0.3:
            return {"kind": "step", "set": "test", "n": _log(rng, 100, 20000), "age": rng.randrange(0, 200)}
        return {"kind": "step", "set": "marun2019", "n": _log(rng, 700, 300000), "age": rng.randrange(0, 400)}
    if kind == "flock":
        if rng.random() < 0.25:
            return {"kind": "flock", "set": "test", "n": _log(rng, 100, 20000), "age": rng.randrange(0, 200),
                    "steps": _log(rng, 1, 100), "forces": rng.random() < 0.3, "pairs": False}
        n = _log(rng, 700, 1 << 20)
        return {"kind": "flock", "set": "marun2019", "n": n, "age": rng.randrange(0, 400),
                "steps": _log(rng, 1, min(100, max(1, 10 * (1 << 20) // n))), "forces": rng.random() < 0.3,
                "pairs": False}
    if kind == "pairs":
        return {"kind": "flock", "set": rng.choice(("marun2019", "test")), "n": _log(rng, 200, 65536),
                "age": rng.randrange(0, 60), "steps": rng.randrange(1, 4), "forces": False, "pairs": True}
    if kind == "sweep":
        low = _log(rng, 700, 2048)
        return {"kind": "sweep", "flocks": _log(rng, 4, 48), "low": low, "high": low + _log(rng, 100, 8000),
                "steps": _log(rng, 20, 200)}
    if kind == "predict":
        return {"kind": "predict", "rows": _log(rng, 1, 65536)}
    return {"kind": "train", "rows": _log(rng, 100, 2048), "epochs": rng.randrange(2, 16),
            "batch": rng.choice((64, 100, 256))}


# ------------------------------------------------------------------ inputs


def _field(case):
    return (case["n"] / SETS[case["set"]][1]) ** (1.0 / 3.0)


def _sim(case, seed, engine="grid", forces=False, pairs=False):
    m, _, placement = SETS[case["set"]]
    sim = B.BoidSimulation(engine, record_forces=forces, allpairs_kernels=pairs)
    sim.setup(case["n"], _field(case), *m["sep"], *m["ali"], *m["coh"], m["vmax"], m["vmin"], placement, seed)
    return sim


def _aged(case, seed):
    """The flock's state `age` updates after its seeded placement, in host memory."""
    with _sim(case, seed) as sim:
        sim.init()
        sim.update(case["age"])
        pos, vel = sim.state()
        return pos.copy(), vel.copy()


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.float32, pin_memory=True).numpy()
    t[:] = a.reshape(-1)
    return t


def _flocks(case, seed):
    """Flocks of the sweep: sizes even over their logarithm, radii, weights and top speed scaled by 0.7 to 1.3."""
    rng = np.random.default_rng(seed)
    m, density, _ = SETS["marun2019"]
    out = []
    for i in range(case["flocks"]):
        n = int(round(math.exp(rng.uniform(math.log(case["low"]), math.log(case["high"])))))
        f = rng.uniform(0.7, 1.3, 7)
        rules = [(m[r][0] * f[j], m[r][1], m[r][2] * f[j + 3]) for j, r in enumerate(("sep", "ali", "coh"))]
        p = B.flock_params(n, (n / density) ** (1.0 / 3.0), *rules, m["vmax"] * f[6], m["vmin"])
        out.append((p, B.INIT_RANDOM_UNIFORM, (seed + 7919 * i) % (1 << 30)))
    return out


def _points(case, seed):
    """Sweep points in the unit cube and smooth, noisy statistics of them."""
    rng = np.random.default_rng(seed)
    x = rng.random((case["rows"], 8), dtype=np.float32)
    w = rng.normal(size=(8, 4))
    t = np.tanh(x @ w - w.sum(0) / 2) + 0.5 * x[:, :4] * x[:, 4:] + 0.05 * rng.normal(size=(case["rows"], 4))
    return x, ((t - t.mean(0)) / (t.std(0) + 1e-12)).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        m, density, _ = SETS[case["set"]]
        pos, vel = (torch.from_numpy(a).cuda() for a in _aged(case, seed))
        return {"kind": kind, "params": B.flock_params(case["n"], _field(case), m["sep"], m["ali"], m["coh"],
                                                       m["vmax"], m["vmin"]),
                "pos": pos, "vel": vel, "pos_out": torch.empty_like(pos), "vel_out": torch.empty_like(vel)}
    if kind == "flock":
        pos, vel = (_pinned(a) for a in _aged(case, seed))
        sim = _sim(case, seed, "allpairs" if case["pairs"] else "grid", case["forces"], case["pairs"])
        return {"kind": kind, "sim": sim, "steps": case["steps"], "forces": case["forces"], "pos": pos, "vel": vel,
                "pos_out": _pinned(np.zeros_like(pos)), "vel_out": _pinned(np.zeros_like(vel))}
    if kind == "sweep":
        return {"kind": kind, "ens": B.Ensemble(_flocks(case, seed)), "steps": case["steps"]}
    x, t = _points(case, seed)
    net = B.Surrogate(8, 256, 4, seed=seed % 1000 + 1)
    if kind == "predict":
        return {"kind": kind, "net": net, "x": x}
    return {"kind": kind, "net": net, "start": net.params(), "x": x, "t": t, "epochs": case["epochs"],
            "batch": case["batch"]}


def run(s):
    kind = s["kind"]
    if kind == "step":
        rc = B.lib().boids_step_noalloc(ctypes.byref(s["params"]), s["pos"].data_ptr(), s["vel"].data_ptr(),
                                        s["pos_out"].data_ptr(), s["vel_out"].data_ptr(),
                                        torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError(B.lib().boids_last_error().decode())
        return [s["pos_out"], s["vel_out"]]
    if kind == "flock":
        sim = s["sim"]
        sim.set_state(s["pos"], s["vel"])
        sim.update(s["steps"])
        out = list(sim.state(s["pos_out"], s["vel_out"]))
        return out + [sim.forces()] if s["forces"] else out
    if kind == "sweep":
        s["ens"].init()
        s["ens"].step(s["steps"])
        return s["ens"].stats()
    if kind == "predict":
        return s["net"].predict(s["x"])
    s["net"].set_params(s["start"])  # also resets the optimiser: every pass is the same fit
    loss = s["net"].train(s["x"], s["t"], epochs=s["epochs"], batch=s["batch"], lr=2e-3, seed=7)
    return [s["net"].params(), loss]


def work(case):
    """Bytes: the state in and out once per update (24 B each way per boid in the caller's layout) and once more
    each way over the host link; the network's rows and parameters.  Operations: 10 per ordered pair of the
    all-pairs kernels, two per multiply-add of the network."""
    kind = case["kind"]
    if kind == "step":
        return {"bytes": 48.0 * case["n"], "flops": 0}
    if kind == "flock":
        n, steps = case["n"], case["steps"]
        return {"bytes": 48.0 * n * (steps + 1) + (36.0 * n if case["forces"] else 0.0),
                "flops": 10.0 * n * n * steps if case["pairs"] else 0}
    if kind == "sweep":
        low, high = case["low"], case["high"]
        mean = (high - low) / math.log(high / low)
        return {"bytes": 48.0 * case["flocks"] * mean * (case["steps"] + 1), "flops": 0}
    macs = 8 * 256 + 256 * 256 + 256 * 4
    if kind == "predict":
        return {"bytes": 48.0 * case["rows"] + 2.0 * macs, "flops": 2.0 * macs * case["rows"]}
    batches = case["epochs"] * -(-case["rows"] // case["batch"])
    return {"bytes": 48.0 * case["rows"] * case["epochs"] + 24.0 * macs * batches,
            "flops": 6.0 * macs * case["rows"] * case["epochs"]}


# ------------------------------------------------------------------ the same in 64 bits


def _update64(pos, vel, case):
    """One update of the flock in 64 bits, every pair that can see each other found directly."""
    m, _, _ = SETS[case["set"]]
    F = _field(case)
    far = max(m["sep"][0], m["ali"][0], m["coh"][0])
    order = torch.argsort(pos[:, 0])
    p, v = pos[order], vel[order]
    n = p.shape[0]
    sums = {r: torch.zeros(n, 3, dtype=torch.float64, device=p.device) for r in ("sep", "ali", "coh")}
    counts = {r: torch.zeros(n, 1, dtype=torch.float64, device=p.device) for r in ("sep", "ali", "coh")}
    speed = v.norm(dim=1)
    rows = 2048
    for i0 in range(0, n, rows):
        pi = p[i0:i0 + rows]
        lo, width = pi[0, 0] - far, pi[-1, 0] - pi[0, 0] + 2 * far
        near = torch.nonzero(torch.remainder(p[:, 0] - lo, F) <= width).squeeze(1)  # the rows' reach along x
        pn = p[near]
        d2 = 0.0
        for c in range(3):
            d = (pn[None, :, c] - pi[:, None, c]).abs()
            d2 = d2 + torch.minimum(d, F - d).square()
        i, j = torch.nonzero(d2 < (far * 1.001) ** 2, as_tuple=True)
        i, j = i + i0, near[j]
        i, j = i[i != j], j[i != j]
        t = p[j]
        t = t - F * (t - p[i] > F / 2).to(t.dtype) + F * (p[i] - t > F / 2).to(t.dtype)  # the nearest image
        r = t - p[i]
        dist = r.norm(dim=1)
        angle = torch.acos(torch.clamp((v[i] * r).sum(1) / (speed[i] * dist), -1.0, 1.0))
        for rule in sums:
            ok = (dist < m[rule][0]) & ((angle <= math.pi * m[rule][1]) | (m[rule][1] >= 1.0))
            what = {"sep": -r / dist[:, None], "ali": v[j], "coh": t}[rule]
            sums[rule].index_add_(0, i[ok], what[ok])
            counts[rule].index_add_(0, i[ok], torch.ones_like(dist[ok])[:, None])
    seen = {r: c > 0 for r, c in counts.items()}
    coh = torch.where(seen["coh"], sums["coh"] / counts["coh"].clamp(min=1) - p, torch.zeros_like(p))
    ali = torch.where(seen["ali"], sums["ali"] / counts["ali"].clamp(min=1) - v, torch.zeros_like(v))
    u = v + m["coh"][2] * coh + m["sep"][2] * sums["sep"] + m["ali"][2] * ali
    s = u.norm(dim=1, keepdim=True)
    u = torch.where(s > m["vmax"], u / s * m["vmax"], torch.where((s > 0) & (s < m["vmin"]), u / s * m["vmin"], u))
    x = p + u
    x = torch.where(x < 0, x + F, torch.where(x > F, x - F, x))
    back = torch.argsort(order)
    return [x[back].cpu(), u[back].cpu()]


def exact(case, seed):
    kind = case["kind"]
    if kind == "predict":
        x, _ = _points(case, seed)
        net = B.Surrogate(8, 256, 4, seed=seed % 1000 + 1)
        p = net.params().astype(np.float64)
        net.close()
        w1, b1, w2, b2, w3, b3 = np.split(p, np.cumsum([8 * 256, 256, 256 * 256, 256, 256 * 4]))
        h = np.maximum(x.astype(np.float64) @ w1.reshape(8, 256) + b1, 0)
        h = np.maximum(h @ w2.reshape(256, 256) + b2, 0)
        return h @ w3.reshape(256, 4) + b3
    # Flocks are chaotic: after several updates a rounding difference has changed who sees whom.  The fit is a
    # long chain of 16-bit roundings in the same way.
    if kind == "step" or (kind == "flock" and case["steps"] == 1 and not case["forces"]):
        pos, vel = (torch.from_numpy(a).cuda().double() for a in _aged(case, seed))
        return _update64(pos, vel, case)
    return None
