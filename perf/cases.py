"""Workloads a user of the particle path runs, as callable cases.

``listed()`` names them, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what a program holds before the call (the initial cloud on
the GPU, a context with its parameters), ``run`` is one pass through the
public API, ``work`` what a pass cannot do without, ``exact`` the same
outputs from plain numpy / torch in 64 bits.

Kinds of case:

* ``steps``  -- load a cloud into a context, advance it, read the state back
  (Simulation.set_particles_device / step / energy / get_particles_device);
* ``sweep``  -- independent trap instances of uneven population stepped
  together (Simulation.batch_set / batch_step);
* ``solver`` -- the stateless solver classes on host arrays, as a host code
  that owns its particles calls them (FastMultipoleSolver, BarnesHutTree);
* ``mlp``    -- the learned correction's network: training, gradients,
  inference on host samples.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "antimatter-kernel_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import amk  # noqa: E402

E = 1.602176634e-19
K_E = 8.9875517923e9
K_B = 1.380649e-23
C_LIGHT = 2.99792458e8
MASS = {"positron": 9.1093837015e-31, "electron": 9.1093837015e-31, "antiproton": 1.67262192369e-27}
SIGN = {"positron": 1.0, "electron": -1.0, "antiproton": -1.0}
MIN_SQ = 1e-30  # pairs closer than this (m^2) are skipped by every solver


def _steps(name, method, n, **over):
    c = {"kind": "steps", "method": method, "n": n, "pair": "positron", "shape": "gaussian", "rx": 1e-4, "rz": 3e-4,
         "temperature": 5.0, "b0": 1.0, "volts": 10.0, "size": 0.01, "steps": 1, "cutoff": 1e-5, "order": 4,
         "theta": 0.5, "leaf": 32, "tensor": False, "learned": False, "cooling": False, "cooling_scale": 1.0,
         "contact": 0.0, "probability": 1.0, "energy_every": 0}
    c.update(over)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # The README run: 100 positrons + 100 electrons, cutoff solver, cooling
        # and annihilation, 100 steps with the energies logged every 10.
        _steps("readme_200", "standard", 200, pair="positron+electron", shape="ellipsoid", rz=1e-4, temperature=1e3,
               steps=100, cooling=True, contact=5e-6, energy_every=10),
        # The same physics for a dense mixed cloud: cutoff cell list, push,
        # contact search, at a size where the kernels count.
        _steps("cutoff_100k", "standard", 100003, pair="positron+electron", shape="ellipsoid", rx=2e-4, rz=2e-4,
               temperature=1e3, steps=10, cutoff=1e-5, cooling=True, contact=2e-6, probability=0.5),
        # Exact all-pairs forces of a positron / antiproton cloud.
        _steps("allpairs_65k", "allpairs", 65536, pair="positron+antiproton", shape="ellipsoid", rx=2e-4, rz=5e-4,
               temperature=10.0, b0=3.0, volts=50.0, steps=4),
        # Barnes-Hut at the comparison's opening angle, an odd count.
        _steps("barnes_hut_524k", "barnes-hut", 524309, theta=0.7, leaf=8),
        # The FMM as params.json gives it by default (order 4, theta 0.5, leaf 32).
        _steps("fmm_p4_262k", "fast-multipole", 262144, pair="positron+electron"),
        # The plain FMM of the one-million comparison.
        _steps("fmm_p6_1m", "fast-multipole", 1048576, order=6),
        # What the autotuner picks for that cloud under 1e-5 (tensor mode).
        _steps("fmm_p7_tensor_1m", "fast-multipole", 1048576, order=7, theta=0.525, leaf=128, tensor=True),
        # Learned p = 2 far field with the network's correction.
        _steps("fmm_learned_200k", "fast-multipole", 200003, order=2, learned=True),
        # The long run at scale: one step of the plain p = 6 FMM with cooling
        # and the annihilation search, positrons and antiprotons.
        _steps("long_4m", "fast-multipole", 4194304, pair="positron+antiproton", shape="ellipsoid", rx=5e-4, rz=2e-3,
               temperature=100.0, b0=5.0, volts=100.0, size=0.02, order=6, cooling=True, cooling_scale=10.0,
               contact=1e-6),
        # A parameter sweep: instances of 100 to 20,000 particles in graph chunks.
        {"name": "sweep_96", "kind": "sweep", "instances": 96, "low": 100, "high": 20000, "steps": 12, "chunk": 5},
        # The solver class on a host code's arrays (copies in and out included).
        {"name": "solver_fmm_20k", "kind": "solver", "what": "fmm", "n": 20011, "order": 4, "theta": 0.5, "leaf": 32},
        # Training the correction's network: Adam on consecutive windows.
        {"name": "mlp_train", "kind": "mlp", "what": "train", "n": 21700, "batch": 4096, "steps": 24},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["cutoff", "cutoff", "allpairs", "barnes-hut", "barnes-hut", "fmm", "fmm", "fmm-tensor",
                       "fmm-tensor", "learned", "sweep", "solver", "mlp"])
    if kind == "cutoff":
        n = _log(rng, 150, 200000)
        r = 1e-4 * rng.uniform(1.0, 3.0)
        near = math.exp(rng.uniform(math.log(0.2), math.log(60.0)))  # mean neighbours within the cutoff
        rc = r * (near / n) ** (1.0 / 3.0)
        return _steps(None, "standard", n, pair="positron+electron", shape="ellipsoid", rx=r, rz=r,
                      temperature=rng.choice([10.0, 1e3]), steps=rng.randint(5, 40), cutoff=rc,
                      cooling=rng.random() < 0.7, contact=rc * rng.uniform(0.1, 0.5),
                      probability=rng.choice([0.5, 1.0]), energy_every=rng.choice([0, 5]))
    if kind == "allpairs":
        n = _log(rng, 500, 65536)
        return _steps(None, "allpairs", n, pair=rng.choice(["positron", "positron+antiproton"]), shape="ellipsoid",
                      rx=2e-4, rz=5e-4, temperature=10.0, b0=3.0, volts=50.0, steps=rng.randint(2, 6))
    if kind == "barnes-hut":
        return _steps(None, "barnes-hut", _log(rng, 2000, 1 << 20), pair=rng.choice(["positron", "positron+electron"]),
                      theta=rng.choice([0.5, 0.7]), leaf=8, tensor=rng.random() < 0.3)
    if kind == "fmm":
        return _steps(None, "fast-multipole", _log(rng, 5000, 1 << 20), order=rng.randint(2, 8),
                      theta=rng.choice([0.4, 0.5, 0.6]), leaf=rng.choice([32, 32, 64]),
                      pair=rng.choice(["positron", "positron+electron"]), shape=rng.choice(["gaussian", "ellipsoid"]))
    if kind == "fmm-tensor":
        return _steps(None, "fast-multipole", _log(rng, 20000, 1 << 20), order=rng.randint(5, 7),
                      theta=rng.choice([0.5, 0.525, 0.55]), leaf=rng.choice([64, 128, 256]), tensor=True,
                      pair=rng.choice(["positron", "positron+antiproton"]))
    if kind == "learned":
        return _steps(None, "fast-multipole", _log(rng, 20000, 400000), order=2, learned=True)
    if kind == "sweep":
        return {"kind": "sweep", "instances": rng.randint(8, 128), "low": rng.randint(64, 300),
                "high": _log(rng, 1000, 20000), "steps": rng.randint(6, 14), "chunk": rng.randint(2, 6)}
    if kind == "solver":
        what = rng.choice(["fmm", "bh"])
        return {"kind": "solver", "what": what, "n": _log(rng, 500, 60000), "order": rng.randint(2, 6),
                "theta": rng.choice([0.5, 0.7]) if what == "bh" else 0.5, "leaf": 8 if what == "bh" else 32}
    what = rng.choice(["train", "train", "gradients", "forward"])
    n = _log(rng, 1000, 60000)
    return {"kind": "mlp", "what": what, "n": n, "batch": min(n, _log(rng, 256, 4096)), "steps": rng.randint(4, 24)}


# ------------------------------------------------------------------ inputs
def _cloud(n, pair, shape, rx, rz, temperature, seed):
    """n particles on the GPU: positions, Maxwellian velocities, species by
    name (equal halves of a pair, first name first)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    d = dict(device="cuda", dtype=torch.float64, generator=g)
    p = torch.randn(3, n, **d)
    if shape == "ellipsoid":
        p = p / p.norm(dim=0) * torch.rand(n, **d).pow(1.0 / 3.0)
    p = p * torch.tensor([rx, rx, rz], device="cuda", dtype=torch.float64)[:, None]
    names = pair.split("+")
    half = n if len(names) == 1 else (n + 1) // 2
    species = torch.full((n,), amk.SPECIES[names[0]], device="cuda", dtype=torch.uint8)
    species[half:] = amk.SPECIES[names[-1]]
    mass = torch.full((n,), MASS[names[0]], device="cuda", dtype=torch.float64)
    mass[half:] = MASS[names[-1]]
    v = torch.randn(3, n, **d) * (K_B * temperature / mass).sqrt()
    sign = torch.full((n,), SIGN[names[0]], device="cuda", dtype=torch.float64)
    sign[half:] = SIGN[names[-1]]
    cols = [p[0], p[1], p[2], v[0], v[1], v[2]]
    return {"x": [c.contiguous() for c in cols], "species": species, "m": mass, "q": sign * E,
            "pops": {names[0]: half} if len(names) == 1 else {names[0]: half, names[1]: n - half}}


def _network(seed):
    """Flat parameters of the 35-128-128-128-3 network (FP32)."""
    g = torch.Generator().manual_seed(int(seed) + 3)
    parts = []
    for out, fan in ((128, 35), (128, 128), (128, 128), (3, 128)):
        parts.append(((torch.rand(out, fan, generator=g) * 2 - 1) * math.sqrt(3.0 / fan)).reshape(-1))
        parts.append(torch.zeros(out))
    return torch.cat(parts).numpy()


def _step_params(c, cl, seed):
    return amk.make_params(
        seed=int(seed) & 0x7FFFFFFF, b0=c["b0"], trap_voltage=c["volts"], z0=c["size"], rho0=c["size"],
        num_steps=max(1, c["steps"]), populations=cl["pops"], temperatures={k: c["temperature"] for k in cl["pops"]},
        cloud_radii=(c["rx"], c["rx"], c["rz"]), bath_temperature=4.0, cooling_scale=c["cooling_scale"],
        cooling_enabled=int(c["cooling"]), coulomb_forces_enabled=1, coulomb_method=c["method"],
        energy_method="standard", cutoff_radius=c["cutoff"], barnes_hut_theta=c["theta"],
        fast_multipole_order=c["order"], fast_multipole_theta=c["theta"], fmm_learned=int(c["learned"]),
        learned_audit_interval=0, annihilation_enabled=int(c["contact"] > 0), contact_radius=c["contact"] or 1e-9,
        annihilation_probability=c["probability"])


def _populations(c):
    m = c["instances"]
    return [int(round(c["low"] * (c["high"] / c["low"]) ** (i / max(1, m - 1)))) for i in range(m)]


def _sweep(c, seed):
    """The instances' clouds and parameters, in order of growing population."""
    rng = random.Random(int(seed))
    clouds, params = [], []
    for i, n in enumerate(_populations(c)):
        pair = rng.choice(["electron+positron", "positron+antiproton"])
        r = math.exp(rng.uniform(math.log(5e-5), math.log(5e-4)))
        temp = math.exp(rng.uniform(math.log(4.0), math.log(1e4)))
        cl = _cloud(n, pair, "ellipsoid", r, r, temp, int(seed) * 1000 + i)
        clouds.append(cl)
        params.append(amk.make_params(
            seed=1 + i, b0=rng.uniform(1.0, 5.0), trap_voltage=rng.uniform(5.0, 50.0), z0=0.01, rho0=0.01,
            num_steps=c["steps"], populations=cl["pops"], temperatures={k: temp for k in cl["pops"]},
            cloud_radii=(r, r, r), bath_temperature=4.0, cooling_scale=1.0, cooling_enabled=1,
            coulomb_forces_enabled=1, coulomb_method="allpairs", energy_method="allpairs", annihilation_enabled=1,
            contact_radius=5e-6, annihilation_probability=0.5))
    return clouds, params


def _samples(c, seed):
    g = torch.Generator().manual_seed(int(seed) + 11)
    x = torch.randn(c["n"], 35, generator=g)
    x[:, 34] = 1.0
    mix = torch.randn(35, 3, generator=g) / math.sqrt(35.0)
    t = torch.sin(x @ mix) + 0.1 * torch.randn(c["n"], 3, generator=g)
    return x.numpy(), t.numpy()


def _host_sources(c, seed):
    cl = _cloud(c["n"], "positron+electron", "gaussian", 1e-4, 3e-4, 5.0, seed)
    return torch.stack(cl["x"][:3], 1).cpu().numpy(), cl["q"].cpu().numpy()


# ------------------------------------------------------------------ the pass
def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "solver":
        pos, q = _host_sources(c, seed)
        cls = amk.FastMultipoleSolver(c["order"], c["theta"], c["leaf"]) if c["what"] == "fmm" else \
            amk.BarnesHutTree(c["theta"], c["leaf"])
        return {"case": c, "pos": pos, "q": q, "solver": cls}
    if c["kind"] == "mlp":
        x, t = _samples(c, seed)
        return {"case": c, "x": x, "t": t, "net": _network(seed), "sim": amk.Simulation()}
    s = {"case": c}
    if c["kind"] == "sweep":
        clouds, s["params"] = _sweep(c, seed)
        s["in"] = [torch.cat([cl["x"][k] for cl in clouds]) for k in range(6)]
        s["species"] = torch.cat([cl["species"] for cl in clouds])
        s["offsets"] = np.concatenate([[0], np.cumsum(_populations(c))])
        s["sim"] = amk.Simulation(s["params"][0])
    else:
        cl = _cloud(c["n"], c["pair"], c["shape"], c["rx"], c["rz"], c["temperature"], seed)
        s["in"], s["species"] = cl["x"], cl["species"]
        sim = s["sim"] = amk.Simulation(_step_params(c, cl, seed))
        sim.set_leaf_sizes(fmm_leaf=c["leaf"] if c["method"] == "fast-multipole" else 32,
                           bh_leaf=c["leaf"] if c["method"] == "barnes-hut" else 8)
        sim.set_fmm_precision("tensor" if c["tensor"] else "fp64")
        if c["learned"]:  # a network trained earlier: its weights replace a token training run's
            torch.cuda.synchronize()
            sim.set_particles_device(c["n"], *[a.data_ptr() for a in s["in"]], s["species"].data_ptr())
            sim.fmm_train_correction(c["theta"], sample_leaves=64, steps=1, batch=32)
            sim.set_mlp_params(_network(seed))
    n = s["species"].numel()
    s["n"] = n
    s["out"] = [torch.empty(n, device="cuda", dtype=torch.float64) for _ in range(6)]
    s["alive"] = torch.empty(n, device="cuda", dtype=torch.uint8)
    torch.cuda.synchronize()  # the clouds are complete before the context's stream reads them
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "solver":
        if c["what"] == "fmm":
            forces, energy = s["solver"].compute(s["pos"], s["q"])
            return {"forces": forces, "energy": np.array([energy])}
        s["solver"].build(s["pos"], s["q"])
        return {"forces": s["solver"].compute_forces()}
    sim = s["sim"]
    if c["kind"] == "mlp":
        sim.set_mlp_params(s["net"])
        if c["what"] == "train":
            loss = sim.mlp_train(s["x"], s["t"], c["steps"], c["batch"], 1e-3)
            return {"params": sim.mlp_params(), "loss": np.array([loss], np.float32)}
        if c["what"] == "gradients":
            loss, grad, y = sim.mlp_gradients(s["x"], s["t"])
            return {"loss": np.array([loss], np.float32), "grad": grad, "y": y}
        return {"y": sim.mlp_forward(s["x"])}
    sim.set_particles_device(s["n"], *[a.data_ptr() for a in s["in"]], s["species"].data_ptr())
    energies = []
    if c["kind"] == "sweep":
        sim.batch_set(s["params"], s["offsets"])
        sim.batch_step(c["steps"], graph_chunk=c["chunk"])
    elif c["energy_every"]:
        for k in range(0, c["steps"], c["energy_every"]):
            sim.step(min(c["energy_every"], c["steps"] - k))
            e = sim.energy()
            energies.append([e["kinetic"], e["trap_potential"], e["coulomb_potential"]])
    else:
        sim.step(c["steps"])
    sim.get_particles_device(*[a.data_ptr() for a in s["out"]], s["alive"].data_ptr())
    out = {"state": s["out"], "alive": s["alive"]}
    if energies:
        out["energies"] = np.array(energies)
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Bytes: every input read once, every output written once, per step. Flops:
    20 per pair the method has to evaluate (all pairs; neighbours within the
    cutoff; for a tree a leaf's 27 neighbours and, per leaf, the 189 cells of
    the classical interaction list through n_m x n_m products; about 200
    monopoles per target in Barnes-Hut); for the network 2 per weight and
    sample forward, 4 more backward."""
    c = dict(case)
    if c["kind"] == "mlp":
        weights = 35 * 128 + 2 * 128 * 128 + 128 * 3
        if c["what"] == "train":
            return {"bytes": 4 * (c["n"] * 38 + 2 * weights), "flops": 6 * weights * c["batch"] * c["steps"]}
        return {"bytes": 4 * c["n"] * 41, "flops": (6 if c["what"] == "gradients" else 2) * weights * c["n"]}
    if c["kind"] == "sweep":
        p = _populations(c)
        return {"bytes": 161 * sum(p) * c["steps"], "flops": 20 * sum(n * n for n in p) * c["steps"]}
    n, steps = c["n"], c.get("steps", 1)
    method = c["method"] if c["kind"] == "steps" else {"fmm": "fast-multipole", "bh": "barnes-hut"}[c["what"]]
    if method == "standard":
        near = min(n, n * (c["cutoff"] / c["rx"]) ** 3)
        flops = 20 * n * near
    elif method == "allpairs":
        flops = 20 * n * n
    elif method == "barnes-hut":
        flops = 20 * n * 200
    else:
        nm = (c["order"] + 1) * (c["order"] + 2) * (c["order"] + 3) // 6
        per_leaf = c["leaf"] / 3.0
        flops = n * (20 * 27 * per_leaf + 189 * 2 * nm * nm / per_leaf + 16 * nm)
    return {"bytes": (161 if c["kind"] == "steps" else 56) * n * steps, "flops": flops * steps}


# ------------------------------------------------------------------ 64-bit values
_PAIRS_LIMIT = 3e11  # pair evaluations of a case that exact() takes on (about 10 s)


def _rows(n):
    return max(1, min(n, (1 << 25) // n))


def _pair_block(x, lo, hi):
    d = [x[k][lo:hi, None] - x[k][None, :] for k in range(3)]
    r2 = d[0] * d[0]
    r2 += d[1] * d[1]
    r2 += d[2] * d[2]
    return d, r2


def _forces(x, q, rc=None):
    """k q_i sum_j q_j r_ij / r^3 over all pairs, or those with r < rc."""
    n = q.numel()
    f = [torch.zeros_like(q) for _ in range(3)]
    for lo in range(0, n, _rows(n)):
        hi = min(n, lo + _rows(n))
        d, r2 = _pair_block(x, lo, hi)
        skip = r2 < MIN_SQ
        if rc is not None:
            skip |= r2 >= rc * rc
        w = r2.masked_fill_(skip, math.inf).pow_(-1.5)
        w *= q[None, :]
        for k in range(3):
            f[k][lo:hi] = K_E * q[lo:hi] * (w * d[k]).sum(1)
    return f


def _potential_energy(x, q, rc=None):
    """Half the sum of k q_i q_j / r (or of the shifted k q_i q_j (1/r - 1/rc) within rc)."""
    n, total = q.numel(), 0.0
    for lo in range(0, n, _rows(n)):
        hi = min(n, lo + _rows(n))
        _, r2 = _pair_block(x, lo, hi)
        skip = r2 < MIN_SQ
        if rc is not None:
            skip |= r2 > rc * rc
        w = r2.rsqrt_() - (0.0 if rc is None else 1.0 / rc)
        w.masked_fill_(skip, 0.0)
        total += float((q[lo:hi, None] * w * q[None, :]).sum())
    return 0.5 * K_E * total


def _philox(k0, k1, c0, c1, c2, c3):
    """Philox4x32-10 (Salmon et al., SC'11): four words per counter, numpy uint64 lanes."""
    m32 = np.uint64(0xFFFFFFFF)
    shape = np.broadcast(c0, c1).shape
    c = [np.broadcast_to(np.asarray(v, np.uint64), shape).copy() for v in (c0, c1, c2, c3)]
    k0, k1 = int(k0), int(k1)
    for _ in range(10):
        a = np.uint64(0xD2511F53) * c[0]
        b = np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & m32, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return [(v.astype(np.float64) + 0.5) * 2.0 ** -32 for v in c]


def _boris(v, f, t, kick_dt, m):
    kick = [fk * (0.5 * kick_dt / m) for fk in f]
    a = [v[k] + kick[k] for k in range(3)]
    p0, p1 = a[0] + a[1] * t, a[1] - a[0] * t
    s = 2.0 * t / (1.0 + t * t)
    return [a[0] + p1 * s + kick[0], a[1] - p0 * s + kick[1], a[2] + kick[2]]


def _push(st, f, p, step, first):
    """Boris push in the trap field, then cyclotron damping and its noise, for the live particles."""
    x, v, q, m, on = st["x"], st["v"], st["q"], st["m"], st["alive"]
    d2 = p.z0 ** 2 / 2.0 + p.rho0 ** 2 / 4.0
    e = [p.trap_voltage / (2 * d2) * x[0], p.trap_voltage / (2 * d2) * x[1], -p.trap_voltage / d2 * x[2]]
    f = [e[k] * q + f[k] for k in range(3)]
    w = list(v)
    if first:
        w = _boris(w, f, -0.5 * p.dt * 0.5 * p.b0 * q / m, -0.5 * p.dt, m)
    w = _boris(w, f, 0.5 * p.dt * p.b0 * q / m, p.dt, m)
    y = [x[k] + w[k] * p.dt for k in range(3)]
    if p.cooling_enabled:
        tau = p.cooling_scale * (0.75 / K_E) * m ** 3 * C_LIGHT ** 3 / (q ** 4 * p.b0 ** 2)
        loss = -torch.expm1(-p.dt / (2 * tau))
        sigma = (K_B * p.bath_temperature / m * loss * (2.0 - loss)).sqrt()
        u = _philox(p.seed, 0xC0011, st["ids"], np.uint64(step), np.uint64(0), np.uint64(0))
        r = np.sqrt(-2.0 * np.log(u[0]))
        for k, trig in ((0, np.cos), (1, np.sin)):
            noise = torch.from_numpy(r * trig(2.0 * np.pi * u[1])).to(w[k].device)
            w[k] = w[k] * (1.0 - loss) + sigma * noise
    for k in range(3):
        x[k] = torch.where(on, y[k], x[k])
        v[k] = torch.where(on, w[k], v[k])


def _annihilate(st, p, step):
    """Contacts of unlike partners matched one at a time in (owner, partner) order."""
    on, sp = st["alive"], st["species"].long()
    kind = torch.where(sp == amk.SPECIES["positron"], 1, torch.where(sp == amk.SPECIES["electron"], -1, 0))
    kind = torch.where(on, kind, 0)
    own, par = [], []
    idx = kind.nonzero().flatten()
    if not (kind == 1).any() or not (kind == -1).any():
        return
    x, kk = [c[idx] for c in st["x"]], kind[idx]
    for lo in range(0, idx.numel(), _rows(idx.numel())):
        hi = min(idx.numel(), lo + _rows(idx.numel()))
        _, r2 = _pair_block(x, lo, hi)
        hit = ((r2 < p.contact_radius ** 2) & (kk[lo:hi, None] * kk[None, :] < 0)).nonzero()
        own.append(idx[hit[:, 0] + lo])
        par.append(idx[hit[:, 1]])
    own, par = torch.cat(own).cpu().numpy(), torch.cat(par).cpu().numpy()
    if not own.size:
        return
    u = _philox(p.seed, 0xA2211, own.astype(np.uint64), par.astype(np.uint64), np.uint64(step), np.uint64(0))[0]
    keep = u < p.annihilation_probability
    own, par = own[keep], par[keep]
    taken = set()
    for k in np.lexsort((par, own)):
        if own[k] not in taken and par[k] not in taken:
            taken.update((int(own[k]), int(par[k])))
    if taken:
        on[torch.tensor(sorted(taken), device=on.device)] = False


def _evolve(cl, p, steps, cutoff, every=0):
    st = {"x": list(cl["x"][:3]), "v": list(cl["x"][3:]), "q": cl["q"], "m": cl["m"], "species": cl["species"],
          "alive": torch.ones_like(cl["q"], dtype=torch.bool), "ids": np.arange(cl["q"].numel(), dtype=np.uint64)}
    energies, before = [], None
    for k in range(1, steps + 1):
        live = torch.where(st["alive"], st["q"], 0.0)
        _push(st, _forces(st["x"], live, cutoff), p, k, k == 1)
        if p.annihilation_enabled:
            _annihilate(st, p, k)
        if every and (k % every == 0 or k == steps):
            live = torch.where(st["alive"], st["q"], 0.0)
            v2 = sum(c * c for c in st["v"])
            kin = float((torch.where(st["alive"], 0.5 * st["m"], 0.0) * v2).sum())
            d2 = p.z0 ** 2 / 2.0 + p.rho0 ** 2 / 4.0
            x = st["x"]
            trap = float((live * p.trap_voltage / (4 * d2) * (2 * x[2] ** 2 - x[0] ** 2 - x[1] ** 2)).sum())
            now = (trap, _potential_energy(x, live, p.cutoff_radius))
            mean = now if before is None else tuple(0.5 * (a + b) for a, b in zip(before, now))
            energies.append([kin, *mean])
            before = now
    return st["x"] + st["v"], energies


def _exact_mlp(c, seed):
    x, t = (torch.from_numpy(a).double().cuda() for a in _samples(c, seed))
    flat = torch.from_numpy(_network(seed)).double().cuda()
    cut, at = [], 0
    for out, fan in ((128, 35), (128, 128), (128, 128), (3, 128)):
        cut += [(at, at + out * fan, (out, fan)), (at + out * fan, at + out * fan + out, (out,))]
        at += out * fan + out

    def forward(flat, x, bf16_inputs=False):
        """The network's outputs and its weights as leaves (matrices rounded to BF16)."""
        leaves, h = [], x
        for k, (lo, hi, shape) in enumerate(cut):
            w = flat[lo:hi].reshape(shape)
            leaves.append((w.float().bfloat16().double() if k % 2 == 0 else w.clone()).requires_grad_())
        for k in range(4):
            h = h @ leaves[2 * k].t() + leaves[2 * k + 1]
            if k < 3:
                h = torch.nn.functional.gelu(h)
        return h, leaves

    def gradients(flat, x, t):
        y, leaves = forward(flat, x)
        loss = ((y - t) ** 2).mean()
        return loss.detach(), torch.cat([g.reshape(-1) for g in torch.autograd.grad(loss, leaves)]), y.detach()

    if c["what"] == "forward":  # the inference path rounds its activations to BF16: no 64-bit value to hold it to
        return None
    if c["what"] == "gradients":
        loss, g, y = gradients(flat, x, t)
        return {"loss": loss.reshape(1), "grad": g, "y": y}
    m, v, loss = torch.zeros_like(flat), torch.zeros_like(flat), None
    batch = min(c["batch"], c["n"])
    for k in range(c["steps"]):
        a = (k * batch) % max(1, c["n"] - batch + 1)
        loss, g, _ = gradients(flat, x[a:a + batch], t[a:a + batch])
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        flat = flat - 1e-3 * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"params": flat, "loss": loss.reshape(1)}


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "mlp":
        return _exact_mlp(c, seed)
    if c["kind"] == "solver":
        pos, q = _host_sources(c, seed)
        x = [torch.from_numpy(np.ascontiguousarray(pos[:, k])).cuda() for k in range(3)]
        q = torch.from_numpy(q).cuda()
        f = torch.stack(_forces(x, q), 1)
        if c["what"] != "fmm":
            return {"forces": f}
        return {"forces": f, "energy": torch.tensor([_potential_energy(x, q)], dtype=torch.float64)}
    if c["kind"] == "sweep":
        if sum(n * n for n in _populations(c)) * c["steps"] > _PAIRS_LIMIT:
            return None
        clouds, params = _sweep(c, seed)
        parts = [_evolve(cl, p, c["steps"], None)[0] for cl, p in zip(clouds, params)]
        return {"state": [torch.cat([s[k] for s in parts]) for k in range(6)], "alive": None}
    if float(c["n"]) ** 2 * c["steps"] > _PAIRS_LIMIT:
        return None
    cl = _cloud(c["n"], c["pair"], c["shape"], c["rx"], c["rz"], c["temperature"], seed)
    state, energies = _evolve(cl, _step_params(c, cl, seed), c["steps"],
                              c["cutoff"] if c["method"] == "standard" else None, c["energy_every"])
    out = {"state": state, "alive": None}
    if energies:
        out["energies"] = np.array(energies)
    return out
