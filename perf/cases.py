"""Performance cases: the work a user of this package has it do.

Every case goes through the public entry points (the Sim and Batch classes,
or the C functions of include/cupic_gpu.h for device and pinned host
buffers).  Kinds of pass:

  cycle    a bias-point run on one context: seeded plasma, `steps` cycles,
           then the potential, field, charge, profiles and counters
  stages   the reference's main loop, one entry point at a time
           (charge_deposition, poisson_solver, field_solver,
           particle_mover, cc)
  batch    many bias-point instances of uneven sizes stepped together
  restart  particles read from host memory, initial mesh, `steps` cycles,
           particles written back to host memory
  poisson  one solve and its field on the caller's device buffers

A pass of the first four starts from its own initial plasma, so that each
does the same work (a fixed number of Jacobi sweeps lets a run of many
hundred steps go unstable).
"""
import ctypes

import numpy as np
import torch

import cupic_gb300 as cg
from cupic_gb300.params import bias_instances, workload_params

LARGE = {"mi": 1836.0, "kti": 0.1, "ds": 0.5, "dt": 0.05, "phi_p": -5.0}


def listed():
    return [
        # the smallest bias-point request, 300 steps alone: launches and latency
        {"name": "cycle_32x128", "kind": "cycle", "ncx": 32, "ncy": 128, "ppc": 30, "sweeps": 200, "steps": 300},
        # the largest size of the bias-point requests
        {"name": "cycle_256x1024", "kind": "cycle", "ncx": 256, "ncy": 1024, "ppc": 30, "sweeps": 200, "steps": 100},
        # the workload at scale, 2.1e8 particles
        {"name": "cycle_512x2048", "kind": "cycle", "ncx": 512, "ncy": 2048, "ppc": 100, "sweeps": 200, "steps": 150},
        # a ragged mesh: rows whose length is no multiple of 4
        {"name": "cycle_301x700", "kind": "cycle", "ncx": 301, "ncy": 700, "ppc": 45, "sweeps": 200, "steps": 60},
        # the small workload: a tolerance tested after every sweep, at most 2000
        {"name": "tol_64x256", "kind": "cycle", "ncx": 64, "ncy": 256, "ppc": 20, "sweeps": 2000, "tol": 1e-6,
         "steps": 40},
        # FP64 potential, corrections every 32 FP32 sweeps
        {"name": "precision_512x2048", "kind": "cycle", "ncx": 512, "ncy": 2048, "ppc": 20, "sweeps": 2000,
         "tol": 1e-10, "refine": 32, "steps": 8},
        # the shipped input file's geometry and stop rule through the stage calls
        {"name": "stages_127x1021", "kind": "stages", "ncx": 127, "ncy": 1021, "ppc": 4, "sweeps": 6000, "tol": 1e-4,
         "steps": 10},
        # the batched form: bias points of 32x128 to 256x1024 cells
        {"name": "batch_64", "kind": "batch", "members": 64, "sweeps": 200, "steps": 80},
        # snapshot in, a few steps, snapshot out
        {"name": "restart_128x512", "kind": "restart", "ncx": 128, "ncy": 512, "ppc": 30, "sweeps": 200, "steps": 20},
        # the solve alone, for callers with their own device buffers
        {"name": "poisson_64x256", "kind": "poisson", "ncx": 64, "ncy": 256, "sweeps": 200},
        {"name": "poisson_250x1000", "kind": "poisson", "ncx": 250, "ncy": 1000, "sweeps": 200},
        {"name": "poisson_512x2048", "kind": "poisson", "ncx": 512, "ncy": 2048, "sweeps": 200},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["cycle", "cycle", "tol", "precision", "stages", "batch", "restart", "poisson", "poisson"])
    if kind == "batch":
        return {"kind": "batch", "members": _log(rng, 4, 64), "sweeps": rng.randint(60, 200),
                "steps": rng.randint(20, 80)}
    ncx = _log(rng, 16, 512)
    if rng.random() < 0.5:
        ncx = max(16, ncx // 4 * 4)
    ncy = min(2048, max(32, int(ncx * rng.uniform(1.0, 6.0))))
    if kind == "poisson":
        return {"kind": "poisson", "ncx": ncx, "ncy": ncy, "sweeps": _log(rng, 20, 400)}
    ppc = _log(rng, 8, 100)
    case = {"kind": "cycle", "ncx": ncx, "ncy": ncy, "ppc": ppc, "sweeps": rng.randint(60, 200),
            "steps": rng.randint(20, 100)}
    if kind == "tol":
        case.update(tol=10.0 ** rng.uniform(-6, -3), sweeps=rng.randint(200, 2000), steps=rng.randint(4, 20))
    elif kind == "precision":
        case.update(tol=10.0 ** rng.uniform(-10, -4), sweeps=rng.randint(300, 2000), refine=rng.choice([16, 32, 50]),
                    steps=rng.randint(2, 8))
    elif kind == "stages":
        case.update(kind="stages", ppc=min(ppc, 20), tol=10.0 ** rng.uniform(-4, -3), sweeps=rng.randint(500, 4000),
                    steps=rng.randint(2, 10))
    elif kind == "restart":
        case.update(kind="restart", ppc=min(ppc, 30), ncx=min(ncx, 256), ncy=min(ncy, 1024),
                    steps=rng.randint(1, 20))
    return case


def _params(case, seed):
    over = dict(LARGE, ncx=case["ncx"], ncy=case["ncy"], seed=seed)
    s, tol, refine = case["sweeps"], case.get("tol", 0.0), case.get("refine", 0)
    if refine:
        over.update(refine_every=refine, tol=tol, min_sweeps=refine, max_sweeps=s, check_every=refine,
                    init_tol=tol, init_min_sweeps=refine, init_max_sweeps=s)
    elif tol > 0:
        # stop rule of the small workload, or of the reference's main loop
        mn = max(case["ncx"], case["ncy"]) + 2 if case["kind"] == "stages" else 1
        over.update(tol=tol, min_sweeps=mn, max_sweeps=s, check_every=1, init_tol=1e-3, init_min_sweeps=mn,
                    init_max_sweeps=s)
        over.update(mi=100.0, kti=1.0)
    else:
        over.update(tol=0.0, min_sweeps=s, max_sweeps=s, check_every=s, init_tol=0.0, init_min_sweeps=s,
                    init_max_sweeps=s)
    if case["kind"] == "stages":
        over.update(ds=0.1, dt=1e-3)
    over["n"] = case.get("ppc", 1) / over["ds"] ** 3
    p = workload_params("large", **over)
    p.eps0 = p.n
    return p.finalize()


def _charge(case, seed):
    """Net charge of a noisy plasma with a sheath, as fixed-point counts."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nny, nnx = case["ncy"] + 1, case["ncx"] + 1
    noise = torch.randn((nny, nnx), generator=g, device="cuda", dtype=torch.float64) * 10.0
    y = torch.arange(nny, device="cuda", dtype=torch.float64)[:, None]
    return torch.round((noise + 20.0 * torch.exp(-y / 8.0)) * 2.0 ** 32).to(torch.int64)


def _linear_phi(p, device):
    j = torch.arange(p.nny, device=device, dtype=torch.float64)[:, None]
    return ((1.0 - j / p.ncy) * p.phi_p).expand(p.nny, p.nnx).contiguous()


def _host_plasma(p, case, seed):
    """A snapshot of both species in pinned host memory."""
    out = []
    for sp, (m, kt) in enumerate(((p.me, p.kte), (p.mi, p.kti))):
        rng = np.random.default_rng([seed, sp])
        n = case["ppc"] * case["ncx"] * case["ncy"]
        buf = torch.empty((n, 4), dtype=torch.float64, pin_memory=True)
        a = buf.numpy()
        a[:, 0] = rng.random(n, dtype=np.float32) * (p.ds * p.ncx) * 0.999999
        a[:, 1] = rng.random(n, dtype=np.float32) * (p.ds * p.ncy) * 0.999999
        a[:, 2:] = rng.standard_normal((n, 2), dtype=np.float32) * np.sqrt(kt / m)
        out.append(buf)
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ps = bias_instances(case["members"], sweeps=case["sweeps"])  # one mix of sizes
        for i, p in enumerate(ps):
            p.seed = 1000 * seed + i
        sims = [cg.Sim(p) for p in ps]
        for s in sims:
            s.init_plasma(wait=False)
        for s in sims:
            s.sync()
        return {"case": case, "sims": sims, "batch": cg.Batch(sims)}
    p = _params(case, seed)
    if kind == "poisson":
        phi0 = _linear_phi(p, "cuda").float()
        return {"case": case, "p": p, "rho": _charge(case, seed), "phi0": phi0, "phi": phi0.clone(),
                "e": torch.zeros((p.nny, p.nnx, 2), device="cuda")}
    st = {"case": case, "p": p, "sim": cg.Sim(p)}
    # a run's particle count is known only after it: snapshot buffers with room
    n = case["ppc"] * case["ncx"] * case["ncy"]
    if kind == "restart":
        st["host"] = _host_plasma(p, case, seed)
        st["out"] = [torch.zeros((n + n // 2 + 4096, 4), dtype=torch.float64).pin_memory() for _ in (0, 1)]
    elif n <= 600000:
        st["out"] = [np.zeros((n + n // 2 + 4096, 4), dtype=np.float32) for _ in (0, 1)]
    return st


def _snapshot(s):
    """Both species into the caller's buffers."""
    for sp, buf in enumerate(s["out"]):
        f32 = isinstance(buf, np.ndarray)
        fn = s["sim"].L.cupic_store_particles_f32 if f32 else s["sim"].L.cupic_store_particles
        ptr = ctypes.cast(buf.ctypes.data if f32 else buf.data_ptr(),
                          ctypes.POINTER(ctypes.c_float if f32 else ctypes.c_double))
        rc = fn(s["sim"].h, sp, ptr, buf.shape[0], ctypes.byref(ctypes.c_int64()))
        if rc:
            raise cg.CupicError(rc, "store_particles")
    return s["out"]


def _read(s):
    """What a user reads after a run."""
    sim, case = s["sim"], s["case"]
    ex, ey = sim.efield()
    st = sim.stats(1)[0]
    out = {"phi": sim.phi(), "ex": ex, "ey": ey, "rho": sim.rho_fixed(),
           "density": [sim.density_profile(0), sim.density_profile(1)],
           "current": sim.probe_current(case["steps"]),
           "counts": list(sim.counts()), "sweeps": st["sweeps"], "residual": st["residual"],
           "absorbed": st["absorbed"], "injected": st["injected"]}
    if "out" in s:
        out["particles"] = _snapshot(s)
    return out


def _run_stages(s):
    sim, p = s["sim"], s["p"]
    t = p.dt
    for _ in range(s["case"]["steps"]):
        sim.charge_deposition()
        sim.poisson_solver(p.tol, min_sweeps=p.min_sweeps, max_sweeps=p.max_sweeps, check_every=1)
        sim.field_solver()
        sim.particle_mover()
        sim.cc(t)
        t += p.dt


def _run_poisson(s):
    p, sweeps = s["p"], s["case"]["sweeps"]
    s["phi"].copy_(s["phi0"])
    done, res = ctypes.c_int32(), ctypes.c_float()
    rc = cg.load_library().cupic_poisson_solver_static(
        ctypes.byref(p), s["rho"].data_ptr(), s["phi"].data_ptr(), s["e"].data_ptr(), 0.0, sweeps, sweeps, sweeps,
        torch.cuda.current_stream().cuda_stream, ctypes.byref(done), ctypes.byref(res))
    if rc:
        raise cg.CupicError(rc, "poisson_solver_static")
    return {"phi": s["phi"], "e": s["e"], "sweeps": done.value, "residual": res.value}


def _run_restart(s):
    sim = s["sim"]
    for sp in (0, 1):
        sim.load(sp, s["host"][sp].numpy())
    sim.init_mesh()
    sim.step(s["case"]["steps"])
    return {"phi": sim.phi(), "rho": sim.rho_fixed(), "particles": _snapshot(s)}


def run(state):
    case = state["case"]
    if case["kind"] == "poisson":
        return _run_poisson(state)
    if case["kind"] == "restart":
        return _run_restart(state)
    if case["kind"] == "batch":
        sims = state["sims"]
        for s in sims:
            s.init_plasma(wait=False)
        for s in sims:
            s.sync()
        state["batch"].step(case["steps"])
        return {"phi": np.concatenate([s.phi().ravel() for s in sims]),
                "rho": np.concatenate([s.rho_fixed().ravel() for s in sims]),
                "counts": np.array([s.counts() for s in sims]),
                "current": np.array([s.probe_current(case["steps"]) for s in sims])}
    state["sim"].init_plasma()
    if case["kind"] == "stages":
        _run_stages(state)
    else:
        state["sim"].step(case["steps"])
    return _read(state)


def work(case):
    """Per cycle: each particle read and written once (32 B), charge, source,
    potential and field of each node once (36 B); per sweep 5 operations a
    node.  The initial plasma is written once and read for its charge."""
    if case["kind"] == "batch":
        shapes = [(p.ncx, p.ncy, p.ppr * p.ncy) for p in bias_instances(case["members"])]
    else:
        shapes = [(case["ncx"], case["ncy"], case.get("ppc", 0) * case["ncx"] * case["ncy"])]
    steps = case.get("steps", 1)
    nbytes = flops = 0.0
    for ncx, ncy, n in shapes:
        nodes = (ncx + 1.0) * (ncy + 1.0)
        nbytes += steps * (2 * n * 32.0 + nodes * 36.0) + 2 * n * 32.0
        flops += steps * (5.0 * nodes * case["sweeps"] + 2 * n * 60.0)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _jacobi64(phi, b, sweeps):
    new = torch.empty_like(phi)
    new.copy_(phi)
    for _ in range(sweeps):
        c = phi[1:-1]
        w = torch.cat([c[:, -2:-1], c[:, :-2]], dim=1)
        new[1:-1, :-1] = 0.25 * ((((b[1:-1, :-1] + w) + c[:, 1:]) + phi[2:, :-1]) + phi[:-2, :-1])
        new[1:-1, -1] = new[1:-1, 0]
        phi, new = new, phi
    return phi, new  # the last two iterates


def _source64(acc, p):
    """acc: charge per node in units of one macroparticle, columns not folded."""
    b = acc.clone()
    b[:, 0] = acc[:, 0] + acc[:, -1]
    b[:, -1] = b[:, 0]
    return b / (p.ds * p.eps0)


def _residual64(phi, b):
    c = phi[1:-1, :-1]
    w = torch.roll(c, 1, 1)
    return (b[1:-1, :-1] - (4.0 * c - (((w + phi[1:-1, 1:]) + phi[2:, :-1]) + phi[:-2, :-1]))).abs().max().item()


def _solve64(phi, b, p, tol, mn, mx):
    if p.refine_every > 0:
        done = 0
        while True:
            if (done >= mn and _residual64(phi, b) < tol) or done >= mx:
                return phi
            k = min(p.refine_every, mx - done)
            phi, _ = _jacobi64(phi, b, k)
            done += k
    if tol <= 0 or mn >= mx:
        return _jacobi64(phi, b, mx)[0]
    done = max(mn - 1, 0)
    phi, _ = _jacobi64(phi, b, done)
    while done < mx:
        phi, old = _jacobi64(phi, b, 1)
        done += 1
        if (phi[1:-1] - old[1:-1]).abs().max().item() < tol:
            break
    return phi


def _field64(phi, ds):
    ex, ey = torch.zeros_like(phi), torch.zeros_like(phi)
    w = torch.cat([phi[:, -2:-1], phi[:, :-2], phi[:, -2:-1]], dim=1)
    e = torch.cat([phi[:, 1:], phi[:, 1:2]], dim=1)
    ex[1:-1] = (w[1:-1] - e[1:-1]) / (2 * ds)
    ey[1:-1] = (phi[:-2] - phi[2:]) / (2 * ds)
    ey[0] = (phi[0] - phi[1]) / ds
    ey[-1] = (phi[-2] - phi[-1]) / ds
    return ex, ey


def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 on int64 tensors of 32-bit words."""
    m, mask = (0xD2511F53, 0xCD9E8D57), 0xFFFFFFFF

    def mul(a, x):  # 32x32 -> (high, low) words without overflow
        lo = (x & 0xFFFF) * a
        hi = (x >> 16) * a + (lo >> 16)
        return hi >> 16, ((hi & 0xFFFF) << 16) | (lo & 0xFFFF)

    k0, k1 = seed & mask, (seed >> 32) & mask
    for _ in range(10):
        h0, l0 = mul(m[0], c0)
        h1, l1 = mul(m[1], c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return [(v.double() + 0.5) * 2.0 ** -32 for v in (c0, c1, c2, c3)]


def _cic(x, y, p):
    sx, sy = x / p.ds, y / p.ds
    i = sx.floor().clamp(0, p.ncx - 1).long()
    j = sy.floor().clamp(0, p.ncy - 1).long()
    return i, j, (sx - i).clamp(0, 1), (sy - j).clamp(0, 1)


def _deposit64(species, p, dev):
    acc = torch.zeros(p.nny * p.nnx, dtype=torch.float64, device=dev)
    for q, (x, y, _, _) in zip((-1.0, 1.0), species):
        i, j, fx, fy = _cic(x, y, p)
        k = i + j * p.nnx
        for dk, w in ((0, (1 - fx) * (1 - fy)), (1, fx * (1 - fy)), (p.nnx, (1 - fx) * fy), (p.nnx + 1, fx * fy)):
            acc.index_add_(0, k + dk, q * w)
    return acc.reshape(p.nny, p.nnx)


def _gather64(x, y, ex, ey, p):
    i, j, fx, fy = _cic(x, y, p)
    k = i + j * p.nnx
    w = (((1 - fx) * (1 - fy), 0), (fx * (1 - fy), 1), ((1 - fx) * fy, p.nnx), (fx * fy, p.nnx + 1))
    fex, fey = ex.reshape(-1), ey.reshape(-1)
    return sum(a * fex[k + d] for a, d in w), sum(a * fey[k + d] for a, d in w)


def _pic64(p, species, steps, start, dev):
    """phi, Ex, Ey of the last of `steps` cycles in 64 bits.  `start`: the
    plasma is a fresh one, whose velocities take half a step back."""
    lx, ly = p.ds * p.ncx, p.ds * p.ncy
    qm = (p.qe / p.me, p.qi / p.mi)
    sig = (np.sqrt(p.kte / p.me), np.sqrt(p.kti / p.mi))
    dtin = [np.sqrt(2.0 * np.pi * m / kt) / (p.n * lx * p.ds) for m, kt in ((p.me, p.kte), (p.mi, p.kti))]
    phi = _solve64(_linear_phi(p, dev), _source64(_deposit64(species, p, dev), p), p, p.init_tol,
                   p.init_min_sweeps, p.init_max_sweeps)
    ex, ey = _field64(phi, p.ds)
    if start:
        for sp in (0, 1):
            x, y, vx, vy = species[sp]
            gx, gy = _gather64(x, y, ex, ey, p)
            species[sp] = (x, y, vx - 0.5 * p.dt * qm[sp] * gx, vy - 0.5 * p.dt * qm[sp] * gy)
    t, tin = p.dt, [p.dt + d for d in dtin]
    for step in range(1, steps + 1):
        phi = _solve64(phi, _source64(_deposit64(species, p, dev), p), p, p.tol, p.min_sweeps, p.max_sweeps)
        ex, ey = _field64(phi, p.ds)
        if step == steps:
            break
        for sp in (0, 1):
            x, y, vx, vy = species[sp]
            gx, gy = _gather64(x, y, ex, ey, p)
            vx, vy = vx + p.dt * qm[sp] * gx, vy + p.dt * qm[sp] * gy
            x, y = torch.remainder(x + p.dt * vx, lx), y + p.dt * vy
            new = [x, y, vx, vy]
            n = 1 + int((t + p.dt - tin[sp]) / dtin[sp]) if tin[sp] < t + p.dt else 0
            if n:
                k = torch.arange(n, device=dev)
                at = tin[sp] + k.double() * dtin[sp]
                tin[sp] += n * dtin[sp]
                z = torch.zeros_like(k)
                u = _philox(k, z + step, z, z + (256 | sp), p.seed)
                ix = u[0] * lx
                ivx = sig[sp] * torch.sqrt(-2.0 * torch.log(u[1])) * torch.cos(2 * np.pi * u[2])
                ivy = -sig[sp] * torch.sqrt(-2.0 * torch.log(u[3]))
                gx, gy = _gather64(ix, torch.full_like(ix, ly), ex, ey, p)
                dp, dv = t + p.dt - at, t + 0.5 * p.dt - at
                inj = [torch.remainder(ix + dp * ivx, lx), ly + dp * ivy, ivx + dv * qm[sp] * gx, ivy + dv * qm[sp] * gy]
                new = [torch.cat(v) for v in zip(new, inj)]
            keep = (new[1] >= 0) & (new[1] < ly)
            species[sp] = tuple(v[keep] for v in new)
        t += p.dt
    return phi, ex, ey


def _plasma64(p, dev):
    out = []
    for sp, s in enumerate((np.sqrt(p.kte / p.me), np.sqrt(p.kti / p.mi))):
        idx = torch.arange(p.ppr * p.ncy, device=dev)
        row = idx // p.ppr
        u = _philox(idx - row * p.ppr, row, torch.zeros_like(idx), torch.zeros_like(idx) + sp, p.seed)
        r = torch.sqrt(-2.0 * torch.log(u[2])) * s
        out.append((u[0] * (p.ds * p.ncx), (row + u[1]) * p.ds, r * torch.cos(2 * np.pi * u[3]),
                    r * torch.sin(2 * np.pi * u[3])))
    return out


def exact(case, seed):
    """The potential and field in 64 bits; counters, fixed-point charge and
    the particles' FP32 state have no such value (a rounding that moves one
    particle across a row shifts the whole list)."""
    kind, dev = case["kind"], "cuda"
    if kind == "batch":
        return None  # minutes of 64-bit cycles
    p = _params(case, seed)
    if kind == "poisson":
        b = _source64(_charge(case, seed).double() * 2.0 ** -32, p)
        phi, old = _jacobi64(_linear_phi(p, dev).float().double(), b, case["sweeps"])
        ex, ey = _field64(phi, p.ds)
        return {"phi": phi, "e": torch.stack([ex, ey], dim=-1), "sweeps": None,
                "residual": (phi[1:-1] - old[1:-1]).abs().max().item()}
    n = 2 * case["ppc"] * case["ncx"] * case["ncy"]
    if n * case["steps"] > 1.2e9 or case["steps"] * case["sweeps"] > 100000 or n > 5e7:
        return None  # over 20 seconds
    if kind == "restart":
        species = []
        for buf in _host_plasma(p, case, seed):
            a = buf.float().double().to(dev)  # the particles as the package stores them
            species.append(tuple(a[:, k].clone() for k in range(4)))
        return {"phi": _pic64(p, species, case["steps"], False, dev)[0]}
    phi, ex, ey = _pic64(p, _plasma64(p, dev), case["steps"], True, dev)
    return {"phi": phi, "ex": ex, "ey": ey}
