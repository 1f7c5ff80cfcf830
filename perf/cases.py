"""What this framework is timed on: the calls its users make, over the sizes they make them at.

Kinds of case (``"do"``):

* ``forward``   the surrogate's inference, ``Mlp.forward``;
* ``train``     one epoch of its training, ``surrogate.train``, and the weights it leaves;
* ``collide``   the allocation-free collision on arrays the caller owns, ``mpcmd_collide_static``;
* ``stages``    the module calls a Fortran driver makes at a collision (distribute, mpc_rotation,
                reaction) and the state they leave in its arrays;
* ``fields``    what a run writes at its output cadence (concentration fields, system series, dimer axes);
* ``period``    one collision period from a host state to a host state (the drop-in boundary);
* ``resident``  one collision period of a run whose state stays on the GPU, with the series it logs;
* ``ensemble``  one collision period of a batch of replicas, with the series it logs.

Whole periods are trajectories: two correct runs differ by rounding, and after a few collisions a particle that
falls into the neighbouring cell in one of them makes that visible.  A ``period`` case therefore starts every pass
from the same host state, and the resident cases return the series a user logs instead of 1.7e8 particles.  Those
have no value in 64 bits short of a second engine, so ``exact`` covers the other kinds.
"""
import math

import numpy as np
import torch

import main_gb300
from main_gb300 import Engine, config, ensemble, surrogate

CUT = 2.0 ** (1.0 / 6.0)


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # the points of a sweep that go back to the network one handful at a time
        dict(name="forward_64", do="forward", rows=64, n_hidden=256, n_layers=4, n_out=2050),
        # a whole sweep in one call: the surrogate's own inference workload
        dict(name="forward_65536", do="forward", rows=65536, n_hidden=256, n_layers=4, n_out=2050),
        # one epoch over the surrogate's 4,096 training replicas at its batch of 256
        dict(name="train_epoch", do="train", points=4096, batch=256, n_hidden=256, n_layers=4, n_out=2050),
        # a host code's own particles, unsorted, in the largest box of this entry point with a round edge
        dict(name="collide_80", do="collide", lx=80, ly=80, lz=80, density=10.0, walls=False, sense=1),
        # the drop-in's collision step on the collective quasi-2D box (z walls)
        dict(name="stages_c1", do="stages", workload="c1", scale=1.0, precision=32),
        # output of a bulk run between two blocks of steps
        dict(name="fields_c2_128", do="fields", workload="c2", scale=0.5, precision=32),
        # the plain single dimer, FP32 and in the FP64 it is specified in
        dict(name="period_c0", do="period", workload="c0", scale=1.0, precision=32),
        dict(name="period_c0_fp64", do="period", workload="c0", scale=1.0, precision=64),
        # the collective quasi-2D box, 64 dimers between walls
        dict(name="period_c1", do="period", workload="c1", scale=1.0, precision=32),
        # the large bulk run: 1.7e8 particles, 512 dimers, Selkov kinetics
        dict(name="resident_c2", do="resident", workload="c2", scale=1.0, precision=32),
        # a small batch (a few points of a sweep) and the ensemble workload
        dict(name="ensemble_16", do="ensemble", replicas=16, edge_lo=16, edge_hi=48, precision=32),
        dict(name="ensemble_256", do="ensemble", replicas=256, edge_lo=16, edge_hi=48, precision=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(("forward", "train", "collide", "stages", "fields", "period", "period", "resident", "ensemble"))
    if do == "forward":
        return dict(do=do, rows=_log_int(rng, 1, 65536), n_hidden=rng.choice((64, 128, 192, 256, 256)),
                    n_layers=rng.randint(1, 6), n_out=rng.choice((2, 35, 514, 2050, 2050)))
    if do == "train":
        return dict(do=do, points=rng.randint(1024, 4096), batch=rng.choice((128, 256, 256, 512)),
                    n_hidden=rng.choice((64, 128, 192, 256, 256)), n_layers=rng.randint(1, 6),
                    n_out=rng.choice((35, 514, 2050, 2050)))
    if do == "collide":
        lx, ly, lz = _log_int(rng, 8, 80), _log_int(rng, 8, 80), _log_int(rng, 8, 79)
        return dict(do=do, lx=lx, ly=ly, lz=lz, density=round(rng.uniform(3.0, 20.0), 2), walls=rng.random() < 0.5,
                    sense=rng.choice((1, -1)))
    if do in ("stages", "fields"):
        w = rng.choice(("c0", "c1", "c2"))
        lo, hi = {"c0": (0.55, 2.0), "c1": (0.25, 1.0), "c2": (0.1, 0.5 if do == "fields" else 0.25)}[w]
        return dict(do=do, workload=w, scale=round(rng.uniform(lo, hi), 3), precision=rng.choice((32, 32, 64)))
    if do == "period":
        w = rng.choice(("c0", "c1", "c2", "rot"))
        lo, hi = {"c0": (0.55, 2.0), "c1": (0.25, 1.0), "c2": (0.1, 0.25), "rot": (0.5, 1.0)}[w]
        return dict(do=do, workload=w, scale=round(rng.uniform(lo, hi), 3), precision=rng.choice((32, 32, 64)))
    if do == "resident":
        return dict(do=do, workload="c2", scale=round(rng.uniform(0.25, 0.75), 3), precision=32)
    lo, fp64 = rng.randint(16, 32), rng.random() < 0.25
    return dict(do=do, replicas=_log_int(rng, 2, 8 if fp64 else 128), edge_lo=lo, edge_hi=rng.randint(lo, 48),
                precision=64 if fp64 else 32)


# ---------------------------------------------------------------- inputs --
def _mlp_params(case, n_in, seed):
    """Weights of a trained network's size (Glorot-uniform, small biases), in the parameter layout of Mlp."""
    rng = np.random.default_rng(seed)
    dims = [n_in] + [case["n_hidden"]] * case["n_layers"] + [case["n_out"]]
    out = []
    for k, n in zip(dims[:-1], dims[1:]):
        a = math.sqrt(6.0 / (n + k))
        out += [rng.uniform(-a, a, n * k), rng.normal(0.0, 0.05, n)]
    return np.concatenate(out).astype(np.float32)


def _train_set(case, seed):
    """Standardised replica parameters and a smooth response of them, with the scatter of a simulated label."""
    rng = np.random.default_rng(seed + 1)
    x = rng.uniform(-1.7, 1.7, (case["points"], surrogate.N_IN)).astype(np.float32)
    g = torch.Generator(device="cuda").manual_seed(seed + 2)
    xd = torch.as_tensor(x, device="cuda")
    a = torch.randn(surrogate.N_IN, 16, generator=g, device="cuda") / 2.0
    b = torch.randn(16, case["n_out"], generator=g, device="cuda") / 4.0
    y = torch.tanh(xd @ a) @ b
    y = y + 0.3 * torch.randn(y.shape, generator=g, device="cuda")
    w = torch.as_tensor(surrogate.output_weights(case["n_out"] - 2), device="cuda")
    return xd, y, w


def _cfg(case, seed):
    return config.workload(case["workload"], scale=case["scale"], precision=case["precision"], seed=seed + 1)


def _pinned_state(n, ns):
    a = {k: torch.empty(n, dtype=torch.float64, pin_memory=True).numpy() for k in ("x", "y", "z", "vx", "vy", "vz")}
    a["flag"] = torch.empty(n, dtype=torch.int32, pin_memory=True).numpy()
    for k in ("dpos", "dvel", "dforce"):
        a[k] = torch.zeros(ns, 3, dtype=torch.float64, pin_memory=True).numpy()
    return a


def _start(case, seed):
    """An engine and the host state of a run in progress: placed by the engine, a tenth of the A particles B."""
    cfg = _cfg(case, seed)
    e = Engine(cfg)
    e.initial()
    st = e.download_state(out=_pinned_state(e.n, max(e.ns, 1)))
    g = torch.Generator(device="cuda").manual_seed(seed + 3)
    turn = (torch.rand(e.n, generator=g, device="cuda") < 0.1).cpu().numpy()
    st["flag"][turn & (st["flag"] == 0)] = 1
    return cfg, e, st


def _collide_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = int(round(case["density"] * case["lx"] * case["ly"] * case["lz"]))
    pos = [torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * case[k] for k in ("lx", "ly", "lz")]
    vel = [torch.randn(n, generator=g, device="cuda", dtype=torch.float64) * math.sqrt(1.0 / 6.0) for _ in range(3)]
    return pos, vel


def _replicas(case, seed):
    return ensemble.sample_replicas(case["replicas"], seed=seed, base_seed=1000 + 7 * seed,
                                    edge=(case["edge_lo"], case["edge_hi"]))


def prepare(case, seed):
    do = case["do"]
    if do == "forward":
        net = surrogate.Mlp(n_hidden=case["n_hidden"], n_layers=case["n_layers"], n_out=case["n_out"],
                            max_rows=max(case["rows"], 128), seed=1)
        net.set_params(_mlp_params(case, net.n_in, seed))
        x = np.random.default_rng(seed + 1).uniform(-1.7, 1.7, (case["rows"], net.n_in)).astype(np.float32)
        return dict(do=do, net=net, x=torch.as_tensor(x, device="cuda"))
    if do == "train":
        net = surrogate.Mlp(n_hidden=case["n_hidden"], n_layers=case["n_layers"], n_out=case["n_out"],
                            batch=case["batch"], max_rows=case["batch"], seed=1)
        net.set_params(_mlp_params(case, net.n_in, seed))
        x, y, w = _train_set(case, seed)
        return dict(do=do, net=net, x=x, y=y, w=w, seed=seed)
    if do == "collide":
        pos, vel = _collide_inputs(case, seed)
        return dict(do=do, pos=pos, vel=vel, step=0, seed=seed, case=case)
    if do == "stages":
        _, e, st = _start(case, seed)
        e.upload_state(st)
        e.prepare()
        return dict(do=do, engine=e, out=_pinned_state(e.n, max(e.ns, 1)))
    if do == "fields":
        cfg, e, st = _start(case, seed)
        e.upload_state(st)
        e.prepare()
        return dict(do=do, engine=e, cfg=cfg)
    if do == "period":
        cfg, e, st = _start(case, seed)
        return dict(do=do, engine=e, cfg=cfg, host=st, out=_pinned_state(e.n, max(e.ns, 1)))
    if do == "resident":
        cfg = _cfg(case, seed)
        e = Engine(cfg)
        e.initial()
        e.prepare()
        return dict(do=do, engine=e, cfg=cfg)
    # (the schedule the autotuner picks for the ensemble workload)
    ens = ensemble.Ensemble(_replicas(case, seed), precision=case["precision"], schedule=(4096, 256, 128))
    ens.initial()
    ens.prepare()
    ens.reset_samples(256)
    return dict(do="ensemble", ens=ens)


# ---------------------------------------------------------------- passes --
def _series(o):
    """One line of the system series, logged in single precision (the FP32 build's sums repeat to rounding)."""
    return [o["kinetic_solvent"], o["kinetic_dimer"], o["potential"]] + [float(v) for v in o["species_count"]]


def run(state):
    do = state["do"]
    if do == "forward":
        return state["net"].forward(state["x"])
    if do == "train":
        losses = surrogate.train(state["net"], state["x"], state["y"], state["w"], epochs=1, seed=state["seed"])
        return {"loss": np.array(losses, dtype=np.float32), "params": state["net"].params()}
    if do == "collide":
        c = state["case"]
        ptr = [t.data_ptr() for t in state["pos"] + state["vel"]]
        status = main_gb300.lib().mpcmd_collide_static(
            *ptr, state["pos"][0].numel(), c["lx"], c["ly"], c["lz"],
            config.GEOM_WALLS if c["walls"] else config.GEOM_PERIODIC, 2.0 * math.pi / 3.0, c["sense"], state["seed"],
            state["step"], torch.cuda.current_stream().cuda_stream)
        if status != 0:
            raise main_gb300.MpcmdError(status, "collide_static")
        state["step"] += 1
        return state["vel"]
    e = state.get("engine")
    if do == "stages":
        e.distribute()
        e.mpc_rotation()
        e.reaction()
        return e.download_state(out=state["out"])
    if do == "fields":
        c = state["cfg"]
        f = e.concentration(0.5 * c["lx"], 0.5 * c["ly"], 0.5 * c["lz"], c["rc"] * CUT)
        o = e.observables()
        f["series"] = np.array([o["kinetic_solvent"]] + [float(v) for v in o["species_count"]], dtype=np.float32)
        f["axes"] = e.dimer_axes(normalize=1)[0]
        return f
    if do == "period":
        e.set_step(0, 0)
        e.upload_state(state["host"])
        e.prepare()
        e.run(state["cfg"]["mpc_every"])
        st = e.download_state(out=state["out"])
        if state["cfg"]["precision"] == 32:
            # sums of single-precision pair forces in no fixed order: a few values that carry no more than that
            st = dict(st, dvel=st["dvel"].astype(np.float32), dforce=st["dforce"].astype(np.float32))
        return st
    if do == "resident":
        e.run(state["cfg"]["mpc_every"])
        axes, speed = e.dimer_axes(normalize=1)
        return {"series": np.array(_series(e.observables()), dtype=np.float32), "axes": axes.astype(np.float32),
                "speed": speed.astype(np.float32)}
    ens = state["ens"]
    ens.run(ens.mpc_every)
    mean, count, axes = ens.samples()
    return {"series": np.array([_series(o) for o in ens.observables()], dtype=np.float32),
            "speed": mean.astype(np.float32), "samples": count, "axes": axes}


# ------------------------------------------------------------------ work --
def _mlp_sizes(case):
    dims = [surrogate.N_IN] + [case["n_hidden"]] * case["n_layers"] + [case["n_out"]]
    weights = sum(a * b for a, b in zip(dims[:-1], dims[1:]))
    return weights, weights + sum(dims[1:])


def _shell(density, rc, rn):
    """Particles between a sphere's surface and its cutoff, both spheres of one dimer: those a step cannot leave out."""
    return density * 4.0 / 3.0 * math.pi * (CUT ** 3 - 1.0) * (rc ** 3 + rn ** 3)


def _period_work(n, cells, shell, steps, real):
    """State (cell, three offsets and velocities, species) read and written once, the shell at every MD step, the
    cell tables once."""
    state = 2 * (5 + 6 * real)
    return n * state + steps * shell * state + cells * 2 * real, n * 60.0 + steps * shell * 80.0


def work(case):
    do = case["do"]
    if do == "forward":
        w, p = _mlp_sizes(case)
        return {"bytes": 4.0 * (case["rows"] * (surrogate.N_IN + case["n_out"]) + p), "flops": 2.0 * case["rows"] * w}
    if do == "train":
        w, p = _mlp_sizes(case)
        rows = case["points"] // case["batch"] * case["batch"]
        # weights and both moments read and written once, the weights and the data
        return {"bytes": 4.0 * (rows * (surrogate.N_IN + case["n_out"]) + 7 * p), "flops": 6.0 * rows * w}
    if do == "collide":
        n = case["density"] * case["lx"] * case["ly"] * case["lz"]
        return {"bytes": 72.0 * n, "flops": 60.0 * n}
    if do == "ensemble":
        b = f = 0.0
        for r in _replicas(case, 1):
            cells = r["lx"] ** 3
            x, y = _period_work(r["n_solvent"], cells, _shell(r["n_solvent"] / cells, r["rc"], r["rn"]), 50,
                                case["precision"] // 8)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    cfg = _cfg(case, 0)
    n, cells, real = cfg["n_solvent"], cfg["lx"] * cfg["ly"] * cfg["lz"], case["precision"] // 8
    host = 52.0 * n
    if do == "stages":      # positions and species in, velocities and species changed, the host arrays written
        return {"bytes": n * (6.0 + 9 * real) + host, "flops": 60.0 * n}
    if do == "fields":
        return {"bytes": n * (5.0 + 6 * real), "flops": 20.0 * n}
    b, f = _period_work(n, cells, cfg["n_dimers"] * _shell(n / cells, cfg["rc"], cfg["rn"]), cfg["mpc_every"], real)
    return {"bytes": b + (2 * host if do == "period" else 0.0), "flops": f}


# ----------------------------------------------------------- in 64 bits --
def _philox(index, extra, step, tag, seed):
    """Philox4x32-10 (Salmon et al., SC'11) of the counters (index, extra, step, tag): two uniforms each."""
    m32 = 0xFFFFFFFF

    def mulhilo(a, b):
        hi = ((a >> 16) * b + (((a & 0xFFFF) * b) >> 16)) >> 16
        return hi & m32, (a * b) & m32

    c = [index.to(torch.int64)] + [torch.full_like(index, v, dtype=torch.int64) for v in (extra, step, tag)]
    k0, k1 = seed & m32, (seed >> 32) & m32
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
        h0, l0 = mulhilo(0xD2511F53, c[0])
        h1, l1 = mulhilo(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
    return [((c[i] << 21) | (c[i + 1] >> 11)).to(torch.float64) * 2.0 ** -53 for i in (0, 2)]


def _collision(pos, vel, lx, ly, lz, walls, angle, sense, seed, step):
    """The stochastic-rotation collision of absolute positions and velocities (CUDA, 64 bits)."""
    zero = torch.zeros(1, dtype=torch.int64, device="cuda")
    u0, u1 = _philox(zero, 0, step, 1, seed)
    u2, _ = _philox(zero, 1, step, 1, seed)
    s = [float(u) - 0.5 for u in (u0, u1, u2)]
    cell = [torch.floor(p) for p in pos]
    off = [p - c for p, c in zip(pos, cell)]
    f = [(torch.remainder(c, L) + torch.floor(o + d)) for c, o, d, L in zip(cell, off, s, (lx, ly, lz))]
    kx, ky = torch.remainder(f[0], lx), torch.remainder(f[1], ly)
    if walls:
        kz = cell[2] + torch.floor(off[2] + s[2] + (1.0 if s[2] < 0 else 0.0))
    else:
        kz = torch.remainder(f[2], lz)
    key = (kx + lx * (ky + ly * kz)).to(torch.int64)
    ncell = lx * ly * (lz + 1 if walls else lz)
    add = lambda v: torch.zeros(ncell, dtype=torch.float64, device="cuda").index_add_(0, key, v)  # noqa: E731
    count = add(torch.ones_like(vel[0])).clamp_(min=1.0)
    cm = [(add(v) / count)[key] for v in vel]
    a0, a1 = _philox(torch.arange(ncell, device="cuda"), 0, step, 2, seed)
    ct = 2.0 * a1 - 1.0
    st = torch.sqrt(1.0 - ct * ct)
    axis = [(st * torch.cos(2.0 * math.pi * a0))[key], (st * torch.sin(2.0 * math.pi * a0))[key], ct[key]]
    d = [v - m for v, m in zip(vel, cm)]
    along = sum(a * q for a, q in zip(axis, d))
    c, sn = math.cos(angle), math.sin(angle) * sense
    out = []
    for i in range(3):
        j, k = (i + 1) % 3, (i + 2) % 3
        out.append(cm[i] + along * axis[i] + c * (d[i] - along * axis[i]) + sn * (axis[j] * d[k] - axis[k] * d[j]))
    return out


def _mlp64(layers, x):
    for i, (w, b) in enumerate(layers):
        x = x @ w.T + b
        if i + 1 < len(layers):
            x = x * torch.sigmoid(x)
    return x


def _layers64(case, flat):
    dims = [surrogate.N_IN] + [case["n_hidden"]] * case["n_layers"] + [case["n_out"]]
    flat, out, at = torch.as_tensor(flat, device="cuda").double(), [], 0
    for k, n in zip(dims[:-1], dims[1:]):
        out.append((flat[at:at + n * k].reshape(n, k).clone(), flat[at + n * k:at + n * k + n].clone()))
        at += n * k + n
    return out


def _train64(case, seed):
    """One epoch of Adam on the weighted squared error, in 64 bits, with the batches of surrogate.train."""
    layers = _layers64(case, _mlp_params(case, surrogate.N_IN, seed))
    p = [t.requires_grad_(True) for pair in layers for t in pair]
    m, v = [torch.zeros_like(t) for t in p], [torch.zeros_like(t) for t in p]
    x, y, w = (t.double() for t in _train_set(case, seed))
    perm = torch.as_tensor(np.random.default_rng(seed).permutation(case["points"]), device="cuda")
    losses = []
    for k, s in enumerate(range(0, case["points"] - case["batch"] + 1, case["batch"])):
        idx = perm[s:s + case["batch"]]
        loss = (w * (_mlp64(list(zip(p[::2], p[1::2])), x[idx]) - y[idx]) ** 2).sum() / case["batch"]
        grads = torch.autograd.grad(loss, p)
        losses.append(float(loss))
        with torch.no_grad():
            for t, g, a, b in zip(p, grads, m, v):
                a.mul_(0.9).add_(0.1 * g)
                b.mul_(0.999).add_(0.001 * g * g)
                t -= 1e-3 * (a / (1 - 0.9 ** (k + 1))) / (torch.sqrt(b / (1 - 0.999 ** (k + 1))) + 1e-8)
    return {"loss": np.array(losses), "params": torch.cat([t.detach().reshape(-1) for t in p])}


def _fields64(cfg, st):
    """output_mod.f95:482-575 of a host state: counts of species A and B in the slabs' bins over the bins' volumes."""
    L = [cfg["lx"], cfg["ly"], cfg["lz"]]
    p = [torch.as_tensor(st[k], device="cuda") for k in ("x", "y", "z")]
    sp = torch.as_tensor(st["flag"], device="cuda")
    nb = [int(v / 0.5) for v in L]
    hw = cfg["rc"] * CUT
    bins = [(torch.ceil(q / 0.5).to(torch.int64) - 1).clamp_(0, n - 1) for q, n in zip(p, nb)]
    inside = [(q - 0.5 * v).abs() <= hw for q, v in zip(p, L)]
    tot = [float((sp == s).sum()) for s in (0, 1)]
    vol = float(L[0] * L[1] * L[2])
    out = {"totals": np.array(tot + [t / vol for t in tot])}
    for s, name in ((0, "a"), (1, "b")):
        for key, i, j, slab in (("c1d", 0, None, 2), ("xy", 0, 1, 2), ("xz", 0, 2, 1), ("yz", 1, 2, 0)):
            at = inside[slab] & (sp == s)
            if j is None:
                c = torch.bincount(bins[i][at], minlength=nb[i]).double() / (0.5 * L[1] * 2.0 * hw)
            else:
                c = torch.bincount((bins[i] + nb[i] * bins[j])[at], minlength=nb[i] * nb[j]).double() / (0.5 * hw)
            out["%s_%s" % (key, name)] = c
    mass = torch.as_tensor(cfg["mass"], dtype=torch.float64, device="cuda")[sp.long()]
    v2 = sum(torch.as_tensor(st[k], device="cuda") ** 2 for k in ("vx", "vy", "vz"))
    kinetic = float((0.5 * mass * v2).sum())
    out["series"] = np.array([kinetic] + [float((sp == s).sum()) for s in range(4)])
    d = st["dpos"][0::2] - st["dpos"][1::2]
    per = (1.0, 1.0, 1.0 if cfg["geometry"] == config.GEOM_PERIODIC else 0.0)
    for c in range(3):
        d[:, c] -= per[c] * L[c] * np.round(d[:, c] / L[c])
    out["axes"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    return out


def exact(case, seed):
    do = case["do"]
    if do == "forward":
        x = np.random.default_rng(seed + 1).uniform(-1.7, 1.7, (case["rows"], surrogate.N_IN)).astype(np.float32)
        with torch.no_grad():
            return _mlp64(_layers64(case, _mlp_params(case, surrogate.N_IN, seed)),
                          torch.as_tensor(x, device="cuda").double())
    if do == "train":
        return _train64(case, seed)
    if do == "collide":
        pos, vel = _collide_inputs(case, seed)
        return _collision(pos, vel, case["lx"], case["ly"], case["lz"], case["walls"], 2.0 * math.pi / 3.0,
                          case["sense"], seed, 0)
    if do == "stages":
        # the arrays in the driver's cell order (a table it holds), a stable sort; the species have no closed value
        cfg, e, st = _start(case, seed)
        order = torch.as_tensor(e.cell_order(), device="cuda").long()
        e.close()
        rank = torch.empty_like(order).index_put_((order,), torch.arange(order.numel(), device="cuda"))
        pos = [torch.as_tensor(st[k], device="cuda") for k in ("x", "y", "z")]
        vel = [torch.as_tensor(st[k], device="cuda") for k in ("vx", "vy", "vz")]
        c = [torch.floor(q).long() for q in pos]
        at = torch.sort(rank[c[0] + cfg["lx"] * (c[1] + cfg["ly"] * c[2])], stable=True).indices
        pos, vel = [q[at] for q in pos], [q[at] for q in vel]
        v = _collision(pos, vel, cfg["lx"], cfg["ly"], cfg["lz"], cfg["geometry"] == config.GEOM_WALLS,
                       cfg["rot_angle"], cfg["rotation_sense"], cfg["seed"], 0)
        return dict(x=pos[0], y=pos[1], z=pos[2], vx=v[0], vy=v[1], vz=v[2])
    if do == "fields":
        cfg, e, st = _start(case, seed)
        e.close()
        return _fields64(cfg, st)
    return None
