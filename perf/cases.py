"""Performance cases: the work a user of the library has it do, through its public entry points.

LJ and SNAP molecular dynamics through the deck driver (`MD`), the host-buffer
step (`MD.run_host`), the force-matching gradient (`fit`) and the batched
ensemble (`Batch`), from a few dozen atoms to LJ-4M.  Starting positions are
lattices with Gaussian displacements and Gaussian velocities, handed to the
driver as a restart file, so every input comes from the seed.

A run ends as a user's program ends it: x, v and f of the owned atoms read
back into page-locked arrays.  The FP64 form's frames stay float64; the mixed
form computes its forces in FP32, and its frames are kept in single precision,
as trajectory files hold them.
"""
from __future__ import annotations

import ctypes
import math
import os
import tempfile

import numpy as np
import torch

import examinimd_gb300 as emd
from examinimd_gb300 import fit

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RHO, LJ_T, CUT, SKIN, EVERY = 0.8442, 1.44, 2.5, 0.3, 20
LJ_A = (4.0 / RHO) ** (1.0 / 3.0)
METAL_BOLTZ, METAL_MVV2E = 8.617343e-5, 1.0364269e-4
SNAP_SETS = {"W": dict(fixture="snap_W_sc", mass=183.84, a_sc=3.1803, a_bcc=3.1803),
             "Ta": dict(fixture="snap_Ta_sc", mass=180.88, a_sc=3.316, a_bcc=3.316)}
# neighbours inside the SNAP cutoff and per LJ row (half of them for a half list)
SNAP_INSIDE, LJ_ROW, LJ_INSIDE = {"bcc": 26, "sc": 18}, 78, 55


def listed():
    return [
        # the smallest deck of the test set: ExaMiniMD's default modules (2D rows, FP64), thermo every 10
        dict(name="lj_deck_864", kind="lj", nx=6, ny=6, nz=6, prec="fp64", neigh="2D", half=False, thermo=10, steps=20),
        # the CPU-sized LJ deck: 32,000 atoms, CSR full list, thermo every 10
        dict(name="lj_deck_32k", kind="lj", nx=20, ny=20, nz=20, prec="fp64", neigh="CSR", half=False, thermo=10,
             steps=20),
        # production-size FP64 drop-in, a ragged box
        dict(name="lj_fp64_913k", kind="lj", nx=61, ny=58, nz=64, prec="fp64", neigh="CSR", half=False, thermo=0,
             steps=20),
        # Newton's third law: half list, newton on, ghost forces folded back
        dict(name="lj_half_144k", kind="lj", nx=33, ny=33, nz=33, prec="fp64", neigh="2D", half=True, thermo=0,
             steps=20),
        # ExaMiniMD's shipped in.lj size (40^3 cells), mixed form, thermo every 10
        dict(name="lj_mixed_256k", kind="lj", nx=40, ny=40, nz=40, prec="mixed", neigh="CSR", half=False, thermo=10,
             steps=20),
        # LJ-4M, the headline deck: five rebuild cycles
        dict(name="lj_mixed_4m", kind="lj", nx=100, ny=100, nz=100, prec="mixed", neigh="CSR", half=False, thermo=0,
             steps=100),
        # the particle state kept in host memory, uploaded and read back every step
        dict(name="lj_host_507k", kind="host", nx=50, ny=47, nz=54, prec="mixed", steps=10),
        # SNAP-W, the headline SNAP deck (mixed form, rebuild every step)
        dict(name="snap_w_mixed_128k", kind="snap", set="W", lattice="bcc", nx=40, ny=40, nz=40, prec="mixed",
             neigh="CSR", thermo=0, steps=2),
        # SNAP W in the FP64 drop-in, a ragged mid-size box, thermo every step
        dict(name="snap_w_fp64_8k", kind="snap", set="W", lattice="bcc", nx=15, ny=17, nz=16, prec="fp64",
             neigh="CSR", thermo=1, steps=2),
        # the shipped in.snap.Ta06A geometry: 64 atoms, 2J = 6, 2D rows
        dict(name="snap_ta_64", kind="snap", set="Ta", lattice="sc", nx=4, ny=4, nz=4, prec="fp64", neigh="2D",
             thermo=0, steps=5),
        # one force-matching gradient: bcc W configurations of uneven size (16 to 1,024 atoms), 56 coefficients
        dict(name="fit_snap_28", kind="fit", configs=28),
        # the batched ensemble: 256 LJ systems of 500 to 20,000 atoms
        dict(name="batch_256", kind="batch", systems=256, steps=500),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _cells(rng, lo, hi, per_cell):
    """Three cell counts near the cube root of a log-uniform atom count."""
    c = (_log(rng, lo, hi) / per_cell) ** (1.0 / 3.0)
    least = math.ceil((lo / per_cell) ** (1.0 / 3.0) - 1e-9)
    return [max(least, round(c * rng.uniform(0.85, 1.18))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["lj64", "lj64", "lj32", "lj32", "host", "snap64", "snap32", "fit", "batch"])
    if kind in ("lj64", "lj32"):
        mixed = kind == "lj32"
        half = rng.random() < 0.25
        nx, ny, nz = _cells(rng, 864, 1.0e6 if mixed else 6.0e5, 4)
        return dict(kind="lj", nx=nx, ny=ny, nz=nz, prec="mixed" if mixed else "fp64",
                    neigh=rng.choice(["CSR", "2D"]), half=half, thermo=0 if half else rng.choice([0, 10]),
                    steps=rng.choice([20, 27, 40]))
    if kind == "host":
        nx, ny, nz = _cells(rng, 4000, 8.0e5, 4)
        return dict(kind="host", nx=nx, ny=ny, nz=nz, prec=rng.choice(["mixed", "mixed", "fp64"]), steps=rng.randint(6, 12))
    if kind in ("snap64", "snap32"):
        mixed = kind == "snap32"
        which, lat = rng.choice(["W", "W", "Ta"]), rng.choice(["bcc", "bcc", "sc"])
        nx, ny, nz = _cells(rng, 128, 60000 if mixed else 12000, 2 if lat == "bcc" else 1)
        return dict(kind="snap", set=which, lattice=lat, nx=nx, ny=ny, nz=nz, prec="mixed" if mixed else "fp64",
                    neigh=rng.choice(["CSR", "2D"]), thermo=0 if mixed else rng.choice([0, 1]), steps=rng.randint(2, 4))
    if kind == "fit":
        return dict(kind="fit", configs=rng.randint(7, 48))
    return dict(kind="batch", systems=int(_log(rng, 8, 200)), steps=rng.choice([60, 100, 200]))


# ---------------------------------------------------------------- inputs from the seed


def _snap_set(name):
    g = np.load(os.path.join(ROOT, "tests", "golden", SNAP_SETS[name]["fixture"] + ".npz"))
    params = {str(k): str(v) for k, v in zip(g["snap_param_keys"], g["snap_param_vals"])}
    return np.array(g["snap_beta"], float), params, SNAP_SETS[name]


def _lattice(style, a, n):
    basis = {"sc": [(0, 0, 0)], "bcc": [(0, 0, 0), (0.5, 0.5, 0.5)],
             "fcc": [(0, 0, 0), (0.5, 0.5, 0), (0.5, 0, 0.5), (0, 0.5, 0.5)]}[style]
    g = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)
    return ((g[:, None, :] + np.asarray(basis)[None]) * a).reshape(-1, 3)


def _particles(case, seed):
    """Positions in [0, box), velocities with no net momentum, box."""
    rng = np.random.default_rng([seed, 1])
    n = [case["nx"], case["ny"], case["nz"]]
    if case["kind"] == "snap":
        s = SNAP_SETS[case["set"]]
        style, a, sigma = case["lattice"], s["a_" + case["lattice"]], 0.05
        vstd = math.sqrt(METAL_BOLTZ * 300.0 / (METAL_MVV2E * s["mass"]))
    else:
        style, a, sigma, vstd = "fcc", LJ_A, 0.04, math.sqrt(LJ_T)
    x = _lattice(style, a, n)
    x += sigma * rng.standard_normal(x.shape)
    box = a * np.asarray(n, float)
    x = np.mod(x, box)
    x[x >= box] = 0.0
    v = vstd * rng.standard_normal(x.shape)
    v -= v.mean(axis=0)
    return x, v, box


def _deck(case, work):
    """The deck a user writes for this case (the restart file brings the atoms)."""
    n = "0 {nx} 0 {ny} 0 {nz}".format(**case)
    if case["kind"] == "snap":
        beta, params, s = _snap_set(case["set"])
        coeff, param = os.path.join(work, "snapcoeff"), os.path.join(work, "snapparam")
        with open(coeff, "w") as fp:
            fp.write("1 %d\n%s 0.5 1\n" % (len(beta), case["set"]) + "".join("%r\n" % float(b) for b in beta))
        with open(param, "w") as fp:
            fp.write("".join("%s %s\n" % kv for kv in params.items()))
        lines = ["units metal", "timestep 0.0005", "atom_style atomic", "newton on",
                 "lattice %s %r" % (case["lattice"], s["a_" + case["lattice"]]), "region box block " + n,
                 "create_box 1 box", "create_atoms 1 box", "mass 1 %r" % s["mass"], "pair_style snap",
                 "pair_coeff * * %s %s %s %s" % (coeff, case["set"], param, case["set"]), "neighbor 1.0 bin",
                 "neigh_modify once no every 1 delay 0 check yes"]
    else:
        lines = ["units lj", "atom_style atomic", "newton %s" % ("on" if case.get("half") else "off"),
                 "lattice fcc %r" % RHO, "region box block " + n, "create_box 1 box", "create_atoms 1 box", "mass 1 1.0",
                 "pair_style lj/cut %r" % CUT, "pair_coeff 1 1 1.0 1.0 %r" % CUT, "neighbor %r bin" % SKIN,
                 "neigh_modify delay 0 every %d check no" % EVERY]
    lines += ["fix 1 all nve", "thermo %d" % case.get("thermo", 0), "run %d" % case["steps"]]
    path = os.path.join(work, "in.deck")
    with open(path, "w") as fp:
        fp.write("\n".join(lines) + "\n")
    return path


def _md(case, seed):
    x, v, _ = _particles(case, seed)
    n = len(x)
    with tempfile.TemporaryDirectory(prefix="emdcase_") as work:
        dump = os.path.join(work, "output.0000000000.000")
        with open(dump, "wb") as fp:
            np.array([n], np.int32).tofile(fp)
            np.arange(1, n + 1, dtype=np.int32).tofile(fp)
            np.zeros(n, np.int32).tofile(fp)
            np.zeros(n).tofile(fp)
            x.tofile(fp)
            v.tofile(fp)
        return emd.MD(["-il", _deck(case, work), "--quiet", "--restart", dump, "--neigh-type", case.get("neigh", "CSR"),
                       "--force-iteration", "NEIGH_HALF" if case.get("half") else "NEIGH_FULL", "--comm-type", "SERIAL",
                       "--precision", case["prec"]])


def _ensemble(case, seed):
    """fcc LJ systems, atom counts log-uniform in [500, 20000]."""
    rng = np.random.default_rng([case["systems"], 2])  # the sizes belong to the case
    target = np.exp(rng.uniform(math.log(500.0), math.log(20000.0), case["systems"]))
    cells = np.maximum(5, np.round((target / 4.0) ** (1.0 / 3.0)).astype(int))
    rng = np.random.default_rng([seed, 2])
    xs, vs, boxes = [], [], []
    for c in cells:
        x = _lattice("fcc", LJ_A, [int(c)] * 3)
        box = np.full(3, c * LJ_A)
        x = np.mod(x + 0.04 * rng.standard_normal(x.shape), box)
        x[x >= box] = 0.0
        v = math.sqrt(LJ_T) * rng.standard_normal(x.shape)
        xs.append(x)
        vs.append(v - v.mean(axis=0))
        boxes.append(box)
    return np.array([len(x) for x in xs]), np.array(boxes), np.concatenate(xs), np.concatenate(vs)


def _fit_inputs(case, seed):
    """Configurations, coefficients and targets: W's coefficients with 5% noise, targets of a shifted set."""
    beta, params, _ = _snap_set("W")
    rng = np.random.default_rng([seed, 3])
    cfgs = fit.snap_config_set(case["configs"], seed=seed)
    n = sum(len(x) for x, _ in cfgs)
    p0 = beta * (1.0 + 0.05 * rng.standard_normal(beta.shape))
    return cfgs, params, p0, rng.normal(0.0, 1.0, len(cfgs)), rng.normal(0.0, 0.5, (n, 3))


# ---------------------------------------------------------------- the cases


def _pinned(n):
    return [torch.empty((n, 3), dtype=torch.float64, pin_memory=torch.cuda.is_available()) for _ in range(3)]


def prepare(case, seed):
    if case["kind"] == "batch":
        n, boxes, x, v = _ensemble(case, seed)
        b = emd.Batch(n, boxes, x, v)
        b.set_shape(1024, 0)  # the form its tuner finds for these ensembles
        return dict(case=case, batch=b)
    if case["kind"] == "fit":
        cfgs, params, p0, e_ref, f_ref = _fit_inputs(case, seed)
        return dict(case=case, configs=[fit.SnapConfig(x, box, params) for x, box in cfgs], p0=torch.tensor(p0),
                    e_ref=torch.tensor(e_ref), f_ref=torch.tensor(f_ref))
    md = _md(case, seed)
    n = md.info()["N_local"]
    st = dict(case=case, md=md, n=n, host=_pinned(n))
    if case["kind"] == "host":
        _read_back(st)  # the host program's arrays, in the driver's order
    return st


def _ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _read_back(st):
    ctx = st["md"].ctx
    x, v, f = st["host"]
    rc = ctx.lib.emd_system_get(ctx.h, 0, st["n"], _ptr(x), _ptr(v), _ptr(f), None, None, None)
    if rc != 0:
        raise RuntimeError("emd_system_get failed")


def run(st):
    case = st["case"]
    if case["kind"] == "batch":
        st["batch"].run(case["steps"])
        return [torch.from_numpy(a).float() for a in st["batch"].get()]
    if case["kind"] == "fit":
        beta = st["p0"].clone().requires_grad_(True)
        energies, forces = fit.SnapEnergyForces.apply(beta, st["configs"])
        fit.loss_fn(energies, forces, st["e_ref"], st["f_ref"], w_E=1e-2, w_F=1.0).backward()
        return dict(E=energies.detach(), F=forces.detach(), grad=beta.grad)
    md = st["md"]
    if case["kind"] == "host":
        md.run_host(case["steps"], *[t.numpy() for t in st["host"]])
    else:
        md.run(case["steps"])
        _read_back(st)
    out = list(st["host"])
    if case.get("thermo"):
        out += [np.float64(t) for t in md.thermo()]
    if case["prec"] == "mixed":
        out = [t.float() if isinstance(t, torch.Tensor) else np.float32(t) for t in out]
    return out


def _snap_terms(J):
    """Terms of the Clebsch-Gordan contraction (half grids of every j1 >= j2, j), elements of the half layers."""
    terms = 0
    for j1 in range(J + 1):
        for j2 in range(j1 + 1):
            for j in range(j1 - j2, min(J, j1 + j2) + 1, 2):
                d = (j1 + j2 - j) // 2
                na = [min(j1, m + d) - max(0, m + d - j2) + 1 for m in range(j + 1)]
                terms += sum(na) * sum(na[: j // 2 + 1])
    return terms, sum((j + 1) * (j // 2 + 1) for j in range(J + 1))


def work(case):
    """Per step: x, v, f of every atom read and written and the neighbour list
    read once; LJ about 23 operations per interacting pair and side; SNAP the
    U sums (8 per element and neighbour), the contraction (8 per term) and the
    pair forces (16 per element and neighbour)."""
    if case["kind"] in ("fit", "snap"):
        if case["kind"] == "fit":
            atoms, lat, J, passes = sum(2 * (2 + k % 7) ** 3 for k in range(case["configs"])), "bcc", 8, 2.0
        else:
            atoms = case["nx"] * case["ny"] * case["nz"] * (2 if case["lattice"] == "bcc" else 1)
            lat, J, passes = case["lattice"], 8 if case["set"] == "W" else 6, float(case["steps"])
        terms, half = _snap_terms(J)
        n = SNAP_INSIDE[lat]
        return dict(bytes=passes * atoms * (144.0 + 8.0 * n), flops=passes * atoms * (24.0 * half * n + 8.0 * terms))
    if case["kind"] == "batch":
        atoms, share, row = case["systems"] * 5300, 1.0, LJ_ROW
    else:
        atoms = 4 * case["nx"] * case["ny"] * case["nz"]
        share = 0.5 if case.get("half") else 1.0
        row = LJ_ROW * share
    return dict(bytes=case["steps"] * atoms * (144.0 + 4.0 * row), flops=case["steps"] * atoms * 23.0 * LJ_INSIDE * share)


# ---------------------------------------------------------------- 64-bit values of the same outputs


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if case["kind"] == "fit":
        return _exact_fit(case, seed, dev) if case["configs"] <= 30 else None
    if case["kind"] == "batch":
        n, boxes, x, v = _ensemble(case, seed)
        if case["systems"] > 40 or n.sum() * case["steps"] > 2.0e7:
            return None
        o = np.concatenate([[0], np.cumsum(n)])
        parts = [_exact_lj(x[o[k]:o[k + 1]], v[o[k]:o[k + 1]], boxes[k], case["steps"], False, dev)
                 for k in range(len(n))]
        return [torch.cat([p[d] for p in parts]) for d in range(3)]
    x, v, box = _particles(case, seed)
    if case["kind"] == "snap":
        if len(x) * case["steps"] > 2.5e4:
            return None
        return _exact_snap(case, x, v, box, dev)
    if len(x) * case["steps"] > 6.0e6 or min(case["nx"], case["ny"], case["nz"]) < 6:
        return None
    out = _exact_lj(x, v, box, case["steps"], True, dev)
    if not case.get("thermo"):
        return out[:3]
    n = len(x)
    mv2 = out[1].square().sum()
    return out[:3] + [np.float64(t) for t in (mv2 / (3 * n - 3), out[3] / n, 0.5 * mv2 / n)]


def _bin_order(x, box, cut):
    """The driver's atom order after a rebuild: bins of at least the list cutoff, x slowest, ascending inside."""
    nb = torch.clamp((box / cut).to(torch.int64), min=1)
    w = box / nb
    nt = nb + 2
    eps = w[0] / 1000
    lo, hi = -w - eps, box + w + eps
    k = ((x - lo) * (nt.double() / (hi - lo))).to(torch.int64)
    return torch.argsort((k[:, 0] * nt[1] + k[:, 1]) * nt[2] + k[:, 2], stable=True)


def _pairs(x, box, cut):
    """Ordered pairs (i, j) closer than `cut` by the minimum image."""
    nb = torch.clamp((box / cut).to(torch.int64), min=1)
    if int(nb.min()) < 3:
        i, j = torch.triu_indices(len(x), len(x), 1, device=x.device)
        d = x[i] - x[j]
        d -= box * torch.round(d / box)
        keep = d.square().sum(1) < cut * cut
        return torch.cat([i[keep], j[keep]]), torch.cat([j[keep], i[keep]])
    c = torch.minimum((x / box * nb).to(torch.int64).clamp(min=0), nb - 1)
    flat = (c[:, 0] * nb[1] + c[:, 1]) * nb[2] + c[:, 2]
    order = torch.argsort(flat)
    count = torch.bincount(flat, minlength=int(nb.prod()))
    start = torch.cumsum(count, 0) - count
    slots = torch.arange(int(count.max()), device=x.device)
    out = []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                o = (c + torch.tensor([dx, dy, dz], device=x.device)) % nb
                f = (o[:, 0] * nb[1] + o[:, 1]) * nb[2] + o[:, 2]
                i, s = torch.nonzero(slots[None] < count[f][:, None], as_tuple=True)
                j = order[start[f[i]] + s]
                d = x[i] - x[j]
                d -= box * torch.round(d / box)
                keep = (d.square().sum(1) < cut * cut) & (i != j)
                out.append((i[keep], j[keep]))
    return torch.cat([p[0] for p in out]), torch.cat([p[1] for p in out])


def _exact_lj(x, v, box, steps, sort, dev):
    x, v = torch.tensor(x, device=dev), torch.tensor(v, device=dev)
    box = torch.tensor(np.asarray(box, float), device=dev)
    cutsq, ecut = CUT * CUT, 4.0 * (CUT ** -12 - CUT ** -6)
    dt = 0.005

    def rebuild(*arrays):
        p = torch.where(arrays[0] < 0, arrays[0] + box, torch.where(arrays[0] > box, arrays[0] - box, arrays[0]))
        o = _bin_order(p, box, CUT + SKIN) if sort else torch.arange(len(p), device=dev)
        return [a[o] for a in (p,) + arrays[1:]] + [_pairs(p[o], box, CUT + SKIN)]

    def force(x, pairs):
        i, j = pairs
        d = x[i] - x[j]
        d -= box * torch.round(d / box)
        r2 = d.square().sum(1)
        inside = r2 < cutsq
        i, d, r2 = i[inside], d[inside], r2[inside]
        s = 1.0 / (r2 * r2 * r2)
        f = torch.zeros_like(x).index_add_(0, i, d * ((48.0 * s - 24.0) * s / r2)[:, None])
        return f, 0.5 * (4.0 * s * (s - 1.0) - ecut).sum()

    x, v, pairs = rebuild(x, v)
    f, pe = force(x, pairs)
    for step in range(1, steps + 1):
        v = v + 0.5 * dt * f
        x = x + dt * v
        if step % EVERY == 0:
            x, v, f, pairs = rebuild(x, v, f)
        f, pe = force(x, pairs)
        v = v + 0.5 * dt * f
    return [x.cpu(), v.cpu(), f.cpu(), float(pe)]


def _cg(j1, j2, j):
    """Clebsch-Gordan coefficients <j1/2 m1 j2/2 m2 | j/2 m> (Racah's formula), zero outside the selection rule."""
    f = math.factorial
    out = np.zeros((j1 + 1, j2 + 1, j + 1))
    delta = math.sqrt(f((j1 + j2 - j) // 2) * f((j1 - j2 + j) // 2) * f((-j1 + j2 + j) // 2) / f((j1 + j2 + j) // 2 + 1))
    for a in range(j1 + 1):
        for b in range(j2 + 1):
            m = a + b - (j1 + j2 - j) // 2
            if not 0 <= m <= j:
                continue
            s = 0.0
            for k in range((j1 + j2) // 2 + j + 2):
                d = [k, (j1 + j2 - j) // 2 - k, j1 - a - k, b - k, (j - j2 + 2 * a - j1) // 2 + k,
                     (j - j1 - 2 * b + j2) // 2 + k]
                if min(d) >= 0:
                    s += (-1) ** k / math.prod(f(q) for q in d)
            out[a, b, m] = s * delta * math.sqrt((j + 1) * f(a) * f(j1 - a) * f(b) * f(j2 - b) * f(m) * f(j - m))
    return out


def _snap_model(params, dev):
    J = int(params["twojmax"])
    rcut, rfac0, rmin0 = float(params["rcutfac"]), float(params["rfac0"]), float(params.get("rmin0", 0))
    triples = [(j1, j2, j) for j1 in range(J + 1) for j2 in range(j1 + 1)
               for j in range(j1 - j2, min(J, j1 + j2) + 1, 2) if j >= j1]
    cg = [torch.tensor(_cg(*t), device=dev, dtype=torch.complex128) for t in triples]

    def u_layers(a, b):
        """Wigner matrices U_j(ma, mb), j = 0..J, of the Cayley-Klein pair (a, b)."""
        u = [torch.ones((len(a), 1, 1), device=dev, dtype=torch.complex128)]
        ac, bc = a.conj()[:, None], b.conj()[:, None]
        for j in range(1, J + 1):
            p = u[-1]
            k = torch.arange(j, device=dev, dtype=torch.float64)
            cols = []
            for mb in range(j):  # U_j(ma, mb) from layer j - 1 for mb < j, the last column by inversion
                lo = torch.sqrt((j - k) / (j - mb)) * ac * p[:, :, mb]
                hi = torch.sqrt((k + 1) / (j - mb)) * bc * p[:, :, mb]
                z = torch.zeros_like(lo[:, :1])
                cols.append(torch.cat([lo, z], 1) - torch.cat([z, hi], 1))
            sign = (-1.0) ** torch.arange(j + 1, device=dev)
            cols.append((sign * cols[0].conj()).flip(1))
            u.append(torch.stack(cols, 2))
        return u

    def bispectrum(x, i, j, box, n):
        """B (n, 55 at 2J = 8) and the repulsion of the pairs, 1.25e5 / r^12 each."""
        d = x[j] - x[i]
        d = d - (box * torch.round(d / box)).detach()
        r2 = d.square().sum(1)
        r = torch.sqrt(r2)
        th = (r - rmin0) * rfac0 * math.pi / (rcut - rmin0)
        s = torch.sin(th) / r
        a = torch.complex(torch.cos(th), -d[:, 2] * s)
        b = torch.complex(d[:, 1] * s, -d[:, 0] * s)
        w = 0.5 * (torch.cos((r - rmin0) * math.pi / (rcut - rmin0)) + 1.0)
        tot = []
        for u in u_layers(a, b):
            k = u.shape[1]
            t = torch.eye(k, device=dev, dtype=torch.complex128).expand(n, k, k)
            tot.append(t.index_add(0, i, u * w[:, None, None]))
        out = []
        for (j1, j2, jj), c in zip(triples, cg):
            # with c real: Z(m, k) = sum c(a, b, m) c(a', b', k) U1(a, a') U2(b, b')
            t = torch.einsum("nxy,xbm->nybm", tot[j1], c)
            t = torch.einsum("nybm,nbz->nymz", t, tot[j2])
            z = torch.einsum("nymz,yzk->nmk", t, c)
            out.append((tot[jj].conj() * z).sum((1, 2)).real)
        return torch.stack(out, 1), 1.25e5 / r2 ** 6

    return rcut, bispectrum


def _exact_snap(case, x, v, box, dev):
    beta, params, s = _snap_set(case["set"])
    rcut, bispectrum = _snap_model(params, dev)
    x, v, box = (torch.tensor(np.asarray(t, float), device=dev) for t in (x, v, box))
    if float(box.min()) < 2.0 * rcut:
        return None
    list_cut = 4.73442 + 1.0  # the deck's pair_style cutoff and skin
    coeff, n = torch.tensor(beta, device=dev), len(x)
    dt, dtfm = 0.0005, 0.5 * 0.0005 / METAL_MVV2E / s["mass"]

    def wrap(x, *rest):
        p = torch.where(x < 0, x + box, torch.where(x > box, x - box, x))
        o = _bin_order(p, box, list_cut)
        return [a[o] for a in (p,) + rest]

    def force(x):
        i, j = _pairs(x, box, rcut)
        x = x.detach().requires_grad_(True)
        b, rep = bispectrum(x, i, j, box, n)
        e = (coeff[0] + b @ coeff[1:]).sum() + rep.sum()
        return -torch.autograd.grad(e, x)[0], float(e.detach())

    x, v = wrap(x, v)
    f, pe = force(x)
    for _ in range(case["steps"]):
        v = v + dtfm * f
        x = x + dt * v
        x, v, f = wrap(x, v, f)
        f, pe = force(x)
        v = v + dtfm * f
    out = [x.cpu(), v.cpu(), f.cpu()]
    if case.get("thermo"):
        mv2 = float(v.square().sum()) * s["mass"]
        out += [np.float64(t) for t in (mv2 * METAL_MVV2E / ((3 * n - 3) * METAL_BOLTZ), pe / n,
                                        0.5 * METAL_MVV2E * mv2 / n)]
    return out


def _exact_fit(case, seed, dev):
    cfgs, params, p0, e_ref, f_ref = _fit_inputs(case, seed)
    rcut, bispectrum = _snap_model(params, dev)
    coeff = torch.tensor(p0, device=dev, requires_grad=True)
    es, fs, loss, o = [], [], 0.0, 0
    grad = torch.zeros_like(coeff)
    n_atoms = sum(len(x) for x, _ in cfgs)
    for k, (x, box) in enumerate(cfgs):
        x = torch.tensor(x, device=dev).requires_grad_(True)
        box = torch.tensor(np.asarray(box, float), device=dev)
        i, j, shift = _image_pairs(x.detach(), box, rcut)
        y = torch.cat([x, x[shift[0]] + shift[1]])
        b, rep = bispectrum(y, i, j, torch.full((3,), 1e6, device=dev, dtype=torch.float64), len(x))
        e = (coeff[0] + b @ coeff[1:]).sum() + rep.sum()
        f = -torch.autograd.grad(e, x, create_graph=True)[0]
        fr = torch.tensor(f_ref[o:o + len(x)], device=dev)
        loss = 1e-2 * (e - e_ref[k]) ** 2 / len(cfgs) + (f - fr).square().sum() / (3 * n_atoms)
        grad += torch.autograd.grad(loss, coeff)[0]
        es.append(float(e.detach()))
        fs.append(f.detach().cpu())
        o += len(x)
    return dict(E=torch.tensor(es, dtype=torch.float64), F=torch.cat(fs), grad=grad.cpu())


def _image_pairs(x, box, cut):
    """Pairs (i, j) within `cut`, j over the atoms and their periodic images (boxes of one to two cutoffs have
    several images of one atom in range): indices into [x, images], and the images' owners and shifts."""
    n, shifts = len(x), []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                if (dx, dy, dz) != (0, 0, 0):
                    shifts.append([dx, dy, dz])
    s = torch.tensor(shifts, device=x.device, dtype=torch.float64) * box
    img = (x[None] + s[:, None]).reshape(-1, 3)
    near = ((img > -cut) & (img < box + cut)).all(1)
    owner = torch.arange(n, device=x.device).repeat(len(shifts))[near]
    y = torch.cat([x, img[near]])
    i, j = torch.nonzero((x[:, None] - y[None]).square().sum(2) < cut * cut, as_tuple=True)
    keep = i != j
    return i[keep], j[keep], (owner, s.repeat_interleave(n, 0)[near])
