"""What a program does with the MD step, as timed cases.

A pass advances a context that the program keeps (`step`, `run` with records), evaluates
forces at the current positions (`forces`), or does a whole short run from host arrays
(`whole`: context, upload, set-up, steps with records, download).  After its steps a pass
reads the state back -- positions, velocities and accelerations -- as a program does that
analyses or stores frames: into pinned host buffers that it keeps.  An FP64 context's
state stays there in FP64; the state of a mixed-precision context, whose forces carry FP32
accuracy, goes on to the GPU as FP32 tensors.

Sizes, densities and parameters are those of the benchmark, the tests and the smoke run
(500 to 4,194,304 atoms, LJ fluid at rho 0.8442, Kob-Andersen mixture, uneven replicas),
with ragged ones between them (vacancies make the atom count odd; boxes with unequal
edges).  Starts are lattices with every atom displaced at random, so that forces are those
of a disordered system from the first step on.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "caviar-v2_gb300"))

import cavgpu  # noqa: E402

BASIS = np.array([[0.0, 0.0, 0.0], [0.5, 0.5, 0.0], [0.5, 0.0, 0.5], [0.0, 0.5, 0.5]])
VV, LANGEVIN, LEAP_FROG = cavgpu.VELOCITY_VERLET, cavgpu.VELOCITY_VERLET_LANGEVIN, cavgpu.LEAP_FROG
FLUID = dict(system="fluid", rho=0.8442, temperature=1.44, skin=0.3, dt=0.005)
MIXTURE = dict(system="mixture", rho=1.2, temperature=0.45, skin=0.3, dt=0.003)
REPLICAS = dict(system="replicas", skin=0.3, dt=0.005)


def listed():
    return [
        # a unit-test-sized system (the smoke run's), every kernel far from filling the GPU
        dict(FLUID, name="step_500_fp64", call="step", nx=5, ny=5, nz=5, vacant=0, precision=0, integrator=VV, steps=20,
             every=0),
        # the reference's ordinary benchmark size, thermo recorded along the way
        dict(FLUID, name="run_4000_mixed", call="run", nx=10, ny=10, nz=10, vacant=0, precision=1, integrator=VV,
             steps=50, every=10),
        # an odd atom count in a box with three different edges; leap-frog, records
        dict(FLUID, name="run_5131_fp64_leapfrog", call="run", nx=13, ny=11, nz=9, vacant=17, precision=0,
             integrator=LEAP_FROG, steps=20, every=5),
        # one Kob-Andersen system under the Langevin thermostat
        dict(MIXTURE, name="step_32000_mixture", call="step", nx=20, ny=20, nz=20, vacant=0, precision=1,
             integrator=LANGEVIN, steps=20, every=0),
        # an ordinary production size in the parity form
        dict(FLUID, name="step_131072_fp64", call="step", nx=32, ny=32, nz=32, vacant=0, precision=0, integrator=VV,
             steps=10, every=0),
        # forces, virial and energy at given positions (a list build each time), ragged
        dict(FLUID, name="forces_255821_mixed", call="forces", nx=41, ny=39, nz=40, vacant=19, precision=1,
             integrator=VV, steps=0, every=0),
        # the headline system, both forms
        dict(FLUID, name="step_1048576_mixed", call="step", nx=64, ny=64, nz=64, vacant=0, precision=1, integrator=VV,
             steps=20, every=0),
        dict(FLUID, name="step_1048576_fp64", call="step", nx=64, ny=64, nz=64, vacant=0, precision=0, integrator=VV,
             steps=10, every=0),
        # the large thermostatted fluid
        dict(FLUID, name="step_4194304_langevin", call="step", nx=128, ny=128, nz=64, vacant=0, precision=1,
             integrator=LANGEVIN, steps=10, every=0, temperature=1.0, skin=0.4),
        # uneven replicas in one context: many (mixed) and few small ones (FP64)
        dict(REPLICAS, name="replicas_256_mixed", call="step", replicas=256, nmin=256, nmax=8192, precision=1,
             integrator=VV, steps=10, every=0),
        dict(REPLICAS, name="replicas_24_fp64", call="step", replicas=24, nmin=256, nmax=2048, precision=0,
             integrator=VV, steps=10, every=0),
        # a whole short run through host memory, every step's thermo read back
        dict(FLUID, name="whole_1048576_mixed", call="whole", nx=64, ny=64, nz=64, vacant=0, precision=1,
             integrator=VV, steps=20, every=1),
    ]


def draw(rng):
    kind = rng.choice(["fluid", "fluid", "fluid", "mixture", "replicas"])
    precision = rng.randint(0, 1)
    if kind == "replicas":
        nmin = int(round(math.exp(rng.uniform(math.log(256), math.log(2048)))))
        nmax = int(round(math.exp(rng.uniform(math.log(nmin + 1), math.log(8192)))))
        most = (1_000_000 if precision else 200_000) // ((nmin + nmax) // 2)
        replicas = int(round(math.exp(rng.uniform(math.log(2), math.log(max(3, min(most, 512)))))))
        return dict(REPLICAS, call="step", replicas=replicas, nmin=nmin, nmax=nmax, precision=precision,
                    integrator=rng.choice([VV, LANGEVIN]), steps=rng.randint(5, 20), every=0)
    call = rng.choice(["step", "step", "run", "forces", "whole"])
    top = 4_000_000 if precision else 1_000_000
    n = math.exp(rng.uniform(math.log(500), math.log(top)))
    edge = (n / 4.0) ** (1.0 / 3.0)
    nx, ny = (max(5, int(round(edge * rng.uniform(0.7, 1.4)))) for _ in range(2))
    nz = max(5, int(round(n / 4.0 / (nx * ny))))
    steps = 0 if call == "forces" else rng.randint(4, 20 if n < 300_000 else 10)
    every = {"run": rng.randint(1, max(1, steps // 2)), "whole": 1}.get(call, 0)
    return dict(FLUID if kind == "fluid" else MIXTURE, call=call, nx=nx, ny=ny, nz=nz, vacant=rng.randint(0, 31),
                precision=precision, integrator=rng.choice([VV, VV, LANGEVIN, LEAP_FROG]), steps=steps, every=every)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _thermal(n, temperature, rng):
    v = rng.normal(0.0, math.sqrt(temperature), size=(n, 3))
    v -= v.mean(0)
    return v * math.sqrt(3 * n * temperature / (v * v).sum())


def _lattice(nx, ny, nz):
    g = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 1, 3)
    return (g + BASIS[None] + 0.25).reshape(-1, 3)


def _inside(pos, box):
    pos = np.mod(pos, box)
    pos[pos >= box] = 0.0  # the remainder of a tiny negative number can round up to the box edge
    return pos


def _systems(case, seed):
    """The case's systems as (pos, vel, type, box) host arrays."""
    rng = np.random.default_rng(seed)
    if case["system"] == "replicas":
        out = []
        sizes = np.random.default_rng([case["replicas"], case["nmin"], case["nmax"]])  # the case's, not the seed's
        for n in sizes.integers(case["nmin"], case["nmax"] + 1, size=case["replicas"]).tolist():
            c = math.ceil((n / 4) ** (1.0 / 3.0))
            box = np.full(3, (n / rng.uniform(0.6, 1.0)) ** (1.0 / 3.0))
            sites = np.sort(rng.choice(4 * c ** 3, size=n, replace=False))
            pos = _lattice(c, c, c)[sites] * (box / c) + rng.uniform(-0.05, 0.05, size=(n, 3))
            out.append((_inside(pos, box), _thermal(n, rng.uniform(0.7, 2.0), rng), np.zeros(n, np.uint64), box))
        return out
    cells = np.array([case["nx"], case["ny"], case["nz"]])
    a = (4.0 / case["rho"]) ** (1.0 / 3.0)
    pos = _lattice(*cells) * a
    if case["vacant"]:
        pos = np.delete(pos, rng.choice(len(pos), size=case["vacant"], replace=False), axis=0)
    n = len(pos)
    typ = np.zeros(n, np.uint64)
    spread = 0.12
    if case["system"] == "mixture":
        typ[rng.permutation(n)[: int(round(0.2 * n))]] = 1
        spread = 0.04
    pos = _inside(pos + rng.uniform(-spread, spread, size=(n, 3)), cells * a)
    return [(pos, _thermal(n, case["temperature"], rng), typ, cells * a)]


def _params(case, box, seed):
    mixture = case["system"] == "mixture"
    eps = np.array([[1.0, 1.5], [1.5, 0.5]]) if mixture else np.ones((1, 1))
    sigma = np.array([[1.0, 0.8], [0.8, 0.88]]) if mixture else np.ones((1, 1))
    rc = 2.5
    return dict(lo=np.zeros(3), hi=box, ntypes=len(eps), nl_cutoff=rc, nl_coef=(rc + case["skin"]) / rc, lj_cutoff=rc,
                eps=eps, sigma=sigma, cutoff_list=2.5 * sigma if mixture else None, mass=np.ones(len(eps)), k_b=1.0,
                dt=case["dt"], integrator=case["integrator"], lang_temperature=case.get("temperature", 1.0),
                lang_friction=1.0, lang_kb=1.0, seed=seed, n_r_df=0 if case["integrator"] == LANGEVIN else 3,
                pressure_process=1)


def _pinned(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def prepare(case, seed):
    systems = _systems(case, seed)
    params = _params(case, systems[0][3], seed)
    n = sum(len(s[0]) for s in systems)
    state = dict(case=case, params=params, n=n, out=[_pinned((n, 3)) for _ in range(3)])
    if case["call"] == "whole":  # host arrays only; the pass does the rest
        pos, vel, typ, _ = systems[0]
        for key, arr, dtype in (("pos", pos, torch.float64), ("vel", vel, torch.float64), ("typ", typ, torch.int64)):
            state[key] = _pinned(arr.shape, dtype).numpy().view(arr.dtype)
            state[key][...] = arr
        return state
    if case["system"] == "replicas":
        md = cavgpu.Batch([(p, v, t, np.zeros(3), b) for p, v, t, b in systems], params, precision=case["precision"])
    else:
        pos, vel, typ, _ = systems[0]
        md = cavgpu.System(pos, vel, typ, params, precision=case["precision"])
    md.setup()
    state["md"] = md
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _read(md, state):
    """Positions, velocities, accelerations through the C ABI into the kept pinned buffers."""
    out = state["out"]
    rc = cavgpu.lib().cavgpu_download(md._h, *(o.data_ptr() for o in out))
    if rc:
        raise cavgpu.CavError(rc, "download")
    return [o.to("cuda").float() for o in out] if state["case"]["precision"] == cavgpu.MIXED else out


def _records(rec, state):
    rec = torch.from_numpy(np.ascontiguousarray(rec))
    return rec.float() if state["case"]["precision"] == cavgpu.MIXED else rec


def run(state):
    case = state["case"]
    if case["call"] == "whole":
        md = cavgpu.System(state["pos"], state["vel"], state["typ"], state["params"], precision=case["precision"])
        md.setup()
        rec = md.run(case["steps"], case["every"])
        pos, vel, acc = _read(md, state)
        md.close()
        return dict(pos=pos, vel=vel, acc=acc, thermo=_records(rec, state))
    md = state["md"]
    if case["call"] == "forces":
        virial, pe = md.forces()
        return dict(acc=_read(md, state)[2], sums=_records(np.array([virial, pe]), state))
    if case["call"] == "run":
        rec = md.run(case["steps"], case["every"])
    else:
        md.step(case["steps"])
        if case["system"] == "replicas":
            rec = md.thermo_batch()[:, :5]
        else:
            t = md.thermo()
            rec = np.array([[t[k] for k in ("ke", "temperature", "pressure", "virial", "pe")]])
    pos, vel, acc = _read(md, state)
    return dict(pos=pos, vel=vel, acc=acc, thermo=_records(rec, state))


def work(case):
    """The state read and written once per step, and every pair inside the cutoff evaluated
    once per step (8 operations for the distance, 11 for the coefficient, 12 to add it to both
    atoms).  A forces pass and a whole run count the evaluation that set-up does, too."""
    if case["system"] == "replicas":
        n, rho = case["replicas"] * (case["nmin"] + case["nmax"]) / 2, 0.8
    else:
        n, rho = 4 * case["nx"] * case["ny"] * case["nz"] - case["vacant"], case["rho"]
    evals = case["steps"] + (case["call"] in ("forces", "whole"))
    pairs = 0.5 * n * rho * 4.0 / 3.0 * math.pi * 2.5 ** 3
    return {"bytes": evals * n * 2 * 9 * 8.0, "flops": evals * pairs * 31.0}


# ---------------------------------------------------------------------------
# the same in plain FP64 torch
# ---------------------------------------------------------------------------
def _pairs_in(pos, box, reach):
    """Every pair within `reach` once: chunks of (i, j, displacement j - i of the nearest image)."""
    n, dev = len(pos), pos.device
    nc = torch.floor(box / reach).long()
    if int(nc.min()) < 3:  # small box: all pairs, nearest image
        i, j = torch.triu_indices(n, n, 1, device=dev)
        for k in range(0, len(i), 1 << 25):
            a, b = i[k:k + (1 << 25)], j[k:k + (1 << 25)]
            d = pos[b] - pos[a]
            d -= torch.round(d / box) * box
            near = (d * d).sum(1) <= reach * reach
            yield a[near], b[near], d[near]
        return
    cell3 = torch.minimum((torch.remainder(pos, box) / box * nc).long(), nc - 1)
    cell = cell3[:, 0] + nc[0] * (cell3[:, 1] + nc[1] * cell3[:, 2])
    order = torch.argsort(cell, stable=True)
    count = torch.bincount(cell, minlength=int(nc.prod()))
    start = torch.cumsum(count, 0) - count
    lanes = torch.arange(int(count.max()), device=dev)
    half = [(x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)][13:]  # the own cell and 13 others
    step = max(1, (1 << 25) // len(lanes))
    for off in half:
        for k in range(0, n, step):
            c = torch.remainder(cell3[k:k + step] + torch.tensor(off, device=dev), nc)
            c = c[:, 0] + nc[0] * (c[:, 1] + nc[1] * c[:, 2])
            a, q = torch.nonzero(lanes[None] < count[c][:, None], as_tuple=True)
            b, a = order[start[c][a] + q], a + k
            if off == (0, 0, 0):
                a, b = a[a < b], b[a < b]
            d = pos[b] - pos[a]
            d -= torch.round(d / box) * box
            near = (d * d).sum(1) <= reach * reach
            yield a[near], b[near], d[near]


def _forces(pos, typ, box, params):
    """Forces, virial sum and potential energy of the shifted-force Lennard-Jones potential."""
    dev = pos.device
    eps, sig = (torch.tensor(params[k], device=dev).reshape(-1) for k in ("eps", "sigma"))
    cut = params["cutoff_list"]
    cut = torch.full_like(eps, params["lj_cutoff"]) if cut is None else torch.tensor(cut, device=dev).reshape(-1)
    s6c = (sig / cut) ** 6
    gc, uc = 4 * eps * s6c * (6 - 12 * s6c) / cut ** 2, 4 * eps * (s6c * s6c - s6c)
    f, virial, pe = torch.zeros_like(pos), 0.0, 0.0
    for a, b, d in _pairs_in(pos, box, float(cut.max())):
        r2 = (d * d).sum(1)
        t = typ[a] * params["ntypes"] + typ[b]
        s6 = (sig[t] ** 2 / r2) ** 3
        inside = r2 <= cut[t] ** 2
        coef = torch.where(inside, 4 * eps[t] * s6 * (6 - 12 * s6) / r2 - gc[t], 0.0)
        pot = 4 * eps[t] * (s6 * s6 - s6) - uc[t] - 0.5 * gc[t] * (r2 - cut[t] ** 2)
        f.index_add_(0, a, coef[:, None] * d)
        f.index_add_(0, b, -coef[:, None] * d)
        virial -= float((coef * r2).sum())
        pe += float(torch.where(inside, pot, 0.0).sum())
    return f, virial, pe


def _noise(seed, step, ids):
    """Three normals per atom from one Philox4x32-10 block, as the Langevin integrator documents them."""
    mask = 0xFFFFFFFF
    c = [torch.full_like(ids, step & mask), torch.full_like(ids, step >> 32), ids, torch.full_like(ids, 0x4C414E47)]
    k0, k1 = seed & mask, seed >> 32

    def mul(m, x):  # 32 x 32 -> 64 bits in halves that fit a signed 64-bit integer
        low = m * (x & 0xFFFF)
        high = m * (x >> 16) + (low >> 16)
        return high >> 16, ((high & 0xFFFF) << 16) | (low & 0xFFFF)

    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    u = [(x.double() + 0.5) * 2.0 ** -32 for x in c]
    r0, r1 = torch.sqrt(-2 * torch.log(u[0])), torch.sqrt(-2 * torch.log(u[2]))
    w = 2 * math.pi
    return torch.stack([r0 * torch.cos(w * u[1]), r0 * torch.sin(w * u[1]), r1 * torch.cos(w * u[3])], 1)


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    got = []
    params = None
    for r, (pos, vel, typ, box) in enumerate(_systems(case, seed)):
        params = params or _params(case, box, seed)  # the replicas share one set of parameters
        x, v = torch.tensor(pos, device=dev), torch.tensor(vel, device=dev)
        t, L, n = torch.tensor(typ.astype(np.int64), device=dev), torch.tensor(box, device=dev), len(pos)
        ids = torch.arange(n, device=dev)
        dt, lang = case["dt"], case["integrator"] == LANGEVIN
        la, lc = (2.0 - dt) / (2.0 + dt), 2.0 * dt / (2.0 + dt)  # friction 1
        lb = math.sqrt(params["lang_temperature"] * 0.5 * dt)
        a, virial, pe = _forces(x, t, L, params)
        rec = [[virial, pe]]
        for k in range(case["steps"]):
            if lang:
                eta = _noise(seed + r, k, ids)
                v = v + 0.5 * dt * a + lb * eta
                mid = v
                x = x + lc * v
            elif case["integrator"] == LEAP_FROG:
                v = v + 0.5 * dt * a
                x = x + dt * v
            else:
                x = x + dt * v + 0.5 * dt * dt * a
            old = a
            a, virial, pe = _forces(x, t, L, params)
            if lang:
                v = la * v + lb * eta + 0.5 * dt * a
            elif case["integrator"] == LEAP_FROG:
                v = v + 0.5 * dt * a
            else:
                v = v + 0.5 * dt * (a + old)
            if k == case["steps"] - 1 or (case["every"] and (k + 1) % case["every"] == 0):
                vt = mid if lang else v  # the Langevin temperature is the mid-step one

                def kinetic(w):
                    return 0.5 * float((w * w).sum() - (0 if lang else (w.sum(0) ** 2).sum() / n))

                # a batch of replicas reports the mid-step kinetic energy, a single system the closing one
                ke_t, ke = kinetic(vt), kinetic(vt if case["system"] == "replicas" else v)
                T = 2 * ke_t / (3 * n - params["n_r_df"])
                vol = float(L.prod())
                rec.append([ke, T, n * T / vol + (0.0 if lang else virial) / (3 * vol), virial, pe])
        x = x - torch.floor(x / L) * L
        got.append((x, v, a, rec))
    if case["call"] == "forces":
        return dict(acc=got[0][2], sums=torch.tensor(got[0][3][0], dtype=torch.float64))
    if case["system"] == "replicas":
        rec = [g[3][-1] for g in got]
    else:
        rec = got[0][3][1:]
        if case["every"]:
            rec = rec[: case["steps"] // case["every"]]
    return dict(zip(("pos", "vel", "acc"), (torch.cat([g[k] for g in got]) for k in range(3))),
                thermo=torch.tensor(rec, dtype=torch.float64))
