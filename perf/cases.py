"""The calls whose speed matters to a user of the framework, with their inputs.

Twelve listed cases and a generator of more of the same ranges.  Each case is
one call (or one short sequence of calls) that a user's program makes through
the Python face of the library:

    df_small, df_full   frequency-shift images of an Fz stack and the gradient
                        back to it (df.df_image_torch): a 64 x 64 thumbnail,
                        where launches and latency count, and the image stack
                        of a full 401 x 401 x 41 scan
    graphene_fp64       Scan.run with its default precision (FP64): the
                        preview a user relaxes first, on a graphene patch
    columns_fp64        Scan.run_columns: a fast run checked in FP64 on pixels
                        spread over the 60-atom cluster
    graphene_df         a whole 101 x 101 x 41 scan of the graphene patch in
                        the executable's default precision (double-float)
    cluster_df          the 60-atom charged cluster, 401 x 401 x 41, the same
    cluster_fast        the same scan in FP32C, the fast path
    batch_fast          run_batch with its default precision (FP32C): 12
                        molecules of 20-400 atoms, points delivered to the host
    slab_df             a periodic 2048-atom slab with an external field:
                        rigid force grid built and relaxed over, double-float
    slab_oneshot        the same kind of slab from scratch in FP32C: field,
                        grid, relaxation, points on the host
    fit_df              one step of fitting a molecule to an image: fz_image,
                        loss, gradients (128 x 128 x 41)
    flex                a flexible molecule, every atom relaxed (FP64)

Sizes are those of the repository's workloads (mechafm_gb300.synth), FP64 and
slab cases on smaller areas.  Points come back as (tip, force, energy, steps,
status) of every record.
"""
import ctypes as C
import math
import os
import tempfile

import numpy as np
import torch

from mechafm_gb300 import _abi, df, synth
from mechafm_gb300.scan import Desc, FlexScan, Input, Scan, run_batch
from mechafm_gb300.torch_ops import fz_image

PREC = {"fp64": _abi.FP64, "fp32c": _abi.FP32C, "df": _abi.DF}


def listed():
    return [
        # a thumbnail's frequency-shift images inside a fitting loop
        dict(name="df_small", kind="df_image", nx=64, ny=64, nz=41, dz=0.1),
        # the image stack of a full-size scan
        dict(name="df_full", kind="df_image", nx=401, ny=401, nz=41, dz=0.1),
        # first look at a new input with the binding's default precision
        dict(name="graphene_fp64", kind="run", system="graphene", precision="fp64", px=51, nz=11,
             step=0.2, atoms=72, integrator="midpoint", minterm="ef"),
        # spot check of a big scan in the reference's arithmetic
        dict(name="columns_fp64", kind="columns", columns=301, px=401, nz=41, step=0.05, atoms=60),
        # an ordinary scan, fewer columns than the GPU has lanes
        dict(name="graphene_df", kind="run", system="graphene", precision="df", px=101, nz=41,
             step=0.1, atoms=72, integrator="midpoint", minterm="ef"),
        # the headline scan
        dict(name="cluster_df", kind="run", system="cluster", precision="df", px=401, nz=41,
             step=0.05, atoms=60, integrator="midpoint", minterm="ef"),
        # the headline scan on the fast path
        dict(name="cluster_fast", kind="run", system="cluster", precision="fp32c", px=401, nz=41,
             step=0.05, atoms=60, integrator="midpoint", minterm="ef"),
        # a data set of small uneven molecules
        dict(name="batch_fast", kind="batch", precision="fp32c", scans=12, small=64, large=128, nz=41),
        # a periodic surface with its Hartree field, grid rebuilt per scan
        dict(name="slab_df", kind="slab", precision="df", px=64, nz=41, fresh=False),
        # the same from the description to the points
        dict(name="slab_oneshot", kind="slab", precision="fp32c", px=97, nz=41, fresh=True),
        # gradient step of a fit
        dict(name="fit_df", kind="fit", precision="df", px=128, nz=41, atoms=60),
        # flexible molecule under the tip
        dict(name="flex", kind="flex", px=5, nz=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["df_image", "run_fp64", "columns", "run_df", "run_df", "run_fp32c", "batch", "slab",
                       "slab", "fit", "flex"])
    integrator = rng.choice(["midpoint", "midpoint", "rk4", "euler"])
    minterm = rng.choice(["ef", "ef", "f", "e"])
    if kind == "df_image":
        return dict(kind=kind, nx=_log_int(rng, 16, 512), ny=_log_int(rng, 16, 401), nz=rng.randint(21, 61),
                    dz=rng.choice([0.05, 0.1, 0.07]))
    if kind.startswith("run_"):
        precision = kind[4:]
        big = precision != "fp64"
        px = _log_int(rng, 21, 301) if big else _log_int(rng, 9, 41)
        return dict(kind="run", system=rng.choice(["graphene", "cluster"]), precision=precision, px=px,
                    nz=rng.randint(11, 41) if big else rng.randint(3, 9), step=rng.choice([0.05, 0.1, 0.2]),
                    atoms=rng.randint(20, 100) if big else rng.randint(20, 72), integrator=integrator,
                    minterm=minterm)
    if kind == "columns":
        return dict(kind=kind, columns=_log_int(rng, 1, 400), px=rng.randint(64, 401), nz=rng.randint(5, 41),
                    step=0.05, atoms=rng.randint(20, 90))
    if kind == "batch":
        return dict(kind=kind, precision=rng.choice(["fp32c", "df"]), scans=rng.randint(2, 12),
                    small=rng.randint(16, 40), large=rng.randint(41, 64), nz=rng.randint(11, 41))
    if kind == "slab":
        fresh = rng.random() < 0.5
        return dict(kind=kind, precision="fp32c" if fresh else "df", px=rng.randint(16, 95 if fresh else 63),
                    nz=rng.randint(11, 41), fresh=fresh)
    if kind == "fit":
        precision = rng.choice(["df", "fp32c", "fp64"])
        px = rng.randint(11, 24) if precision == "fp64" else _log_int(rng, 24, 128)
        nz = rng.randint(3, 7) if precision == "fp64" else rng.randint(11, 41)
        return dict(kind=kind, precision=precision, px=px, nz=nz, atoms=rng.randint(20, 90))
    return dict(kind="flex", px=rng.randint(1, 7), nz=rng.randint(2, 6))


# ---- inputs -----------------------------------------------------------------

def _zlow(zhigh, dz, nz):
    """The lowest height of nz levels, a hair below the last one (the level count is rounded down)."""
    return round(zhigh - dz * (nz - 1) - 1e-6, 9)


def _load(spec):
    with tempfile.TemporaryDirectory() as tmp:
        return Input(spec.write(os.path.join(tmp, spec.name)))


def _scan_spec(case, seed):
    """A scan's input: a graphene patch with thermal displacements, or the charged cluster."""
    kw = dict(area=(case["px"] - 1) * case["step"], step=case["step"], zhigh=10.0,
              zlow=_zlow(10.0, 0.1, case["nz"]), dz=0.1)
    for key in ("integrator", "minterm"):
        if key in case:
            kw[key] = case[key]
    if case.get("system", "cluster") == "cluster":
        return synth.cluster_60(seed=seed, n_atoms=case["atoms"], **kw)
    spec = synth.graphene_72(**kw)
    rng = np.random.default_rng(seed)
    spec.pos = spec.pos + rng.normal(0.0, 0.02, spec.pos.shape)
    return spec


def _device_points(n):
    return torch.empty(n, 8, dtype=torch.float64, device="cuda")


def _point_parts(p):
    """(tip, force, energy, steps, status) of the records, as views."""
    if isinstance(p, torch.Tensor):
        i = p.view(torch.int32)
        return {"tip": p[:, 0:3], "force": p[:, 3:6], "energy": p[:, 6], "steps": i[:, 14], "status": i[:, 15]}
    return {"tip": p["tip"], "force": p["force"], "energy": p["energy"], "steps": p["steps"],
            "status": p["status"]}


def _flex_input(case, seed):
    return _load(synth.flexible_naphthalene(seed=seed, area=0.5 * (case["px"] - 1), step=0.5, zhigh=10.0,
                                            zlow=_zlow(10.0, 0.2, case["nz"]), dz=0.2))


def _slab_desc(case, seed):
    """The 2048-atom periodic slab and, as a program that has it in memory hands it over, its Hartree
    potential on 160 x 160 x 120 voxels (in the scan's energy unit, kcal/mol)."""
    spec = synth.slab(seed=seed, pixels=case["px"], zhigh=18.0, zlow=_zlow(18.0, 0.1, case["nz"]),
                      external=False, tip_charge=-0.02)
    rng = np.random.default_rng(seed)
    base = _load(spec).desc()
    n, cell = (160, 160, 120), (40.0, 40.0, 30.0)
    pot = synth.gaussian_potential(spec.pos, rng.normal(0.0, 0.3, len(spec.pos)), np.diag(cell), n) * -627.50961
    c = _abi.ScanDesc.from_buffer_copy(base.c)
    c.use_external_potential = 1
    c.epot = pot.ctypes.data_as(C.POINTER(C.c_double))
    for k in range(3):
        c.epot_n[k] = n[k]
        c.epot_origin[k] = base.c.offset[k]
        for m in range(3):
            c.epot_basis[3 * k + m] = cell[k] / n[k] if k == m else 0.0
    return Desc(c, keep=(base, pot))


def _fz_stack(case, seed):
    """An Fz stack as a scan leaves it: attraction that grows towards the surface, with contrast in x and y."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.rand(4, generator=g, device="cuda", dtype=torch.float64)
    x = torch.arange(case["nx"], device="cuda", dtype=torch.float64)[:, None, None] * 0.05
    y = torch.arange(case["ny"], device="cuda", dtype=torch.float64)[None, :, None] * 0.05
    z = torch.arange(case["nz"], device="cuda", dtype=torch.float64)[None, None, :] * case["dz"]
    fz = -0.05 * torch.exp(0.9 * z) * (1 + 0.3 * torch.cos(2.5 * x + 6 * r[0]) * torch.cos(2.1 * y + 6 * r[1]))
    fz = fz + 0.002 * torch.exp(1.6 * z) * (1 + 0.2 * torch.sin((1 + r[2]) * x + y))
    return fz + 1e-4 * torch.randn(fz.shape, generator=g, device="cuda", dtype=torch.float64)


def _target(case, seed):
    """A measured image stack to fit: smooth contrast plus noise."""
    rng = np.random.default_rng(seed + 1)
    n, nz = case["px"], case["nz"]
    a = rng.uniform(0.5, 1.5, 3)
    x = np.arange(n)[:, None, None] * 0.1
    y = np.arange(n)[None, :, None] * 0.1
    z = np.arange(nz)[None, None, :] * 0.1
    t = -0.02 * np.exp(0.6 * z) * (1 + 0.3 * np.cos(a[0] * x + a[2]) * np.cos(a[1] * y))
    return torch.from_numpy(t + rng.normal(0.0, 1e-3, t.shape))


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "df_image":
        s["fz"] = _fz_stack(case, seed).requires_grad_(True)
        nw = len(df.weights(case["dz"])[0])
        g = torch.Generator(device="cuda").manual_seed(seed + 7)
        s["grad"] = torch.randn(case["nz"] - nw, case["nx"], case["ny"], generator=g, device="cuda",
                                dtype=torch.float64)
    elif kind in ("run", "columns"):
        desc = _load(_scan_spec(case, seed)).desc()
        s["scan"] = Scan(desc, device=0)
        if kind == "columns":
            rng = np.random.default_rng(seed)
            s["columns"] = np.sort(rng.choice(desc.n_columns, case["columns"], replace=False)).astype(np.int32)
        elif case["precision"] != "fp64":
            s["out"] = _device_points(desc.n_points)
    elif kind == "batch":
        zlow = _zlow(10.0, 0.1, case["nz"])
        specs = [synth.molecule_batch(1, seed=12 * seed + k, grids=(case["large" if k % 2 else "small"],), zlow=zlow)[0]
                 for k in range(case["scans"])]
        s["scans"] = [Scan(_load(p).desc(), device=0) for p in specs]
    elif kind == "slab":
        desc = _slab_desc(case, seed)
        s["desc"] = desc
        if not case["fresh"]:
            s["scan"] = Scan(desc, device=0)
            s["out"] = _device_points(desc.n_points)
    elif kind == "fit":
        sc = dict(case, system="cluster", step=0.1)
        desc = _load(_scan_spec(sc, seed)).desc()
        a = desc.atoms()
        s["desc"] = desc
        s["theta"] = [torch.tensor(v, dtype=torch.float64, requires_grad=True)
                      for v in (a["pos"], a["charge"], desc.pair_params())]
        s["target"] = _target(case, seed)
    elif kind == "flex":
        inp = _flex_input(case, seed)
        s["scan"] = FlexScan(inp.desc(), inp.flex_desc(), device=0)
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "df_image":
        img = df.df_image_torch(s["fz"], case["dz"])
        (g,) = torch.autograd.grad(img, s["fz"], s["grad"])
        return {"df": img.detach(), "dfz": g}
    if kind == "run":
        if case["precision"] == "fp64":
            pts, _ = s["scan"].run()
            return _point_parts(pts)
        s["scan"].run_device(s["out"].data_ptr(), PREC[case["precision"]])
        return _point_parts(s["out"])
    if kind == "columns":
        pts, _ = s["scan"].run_columns(s["columns"])
        return _point_parts(pts)
    if kind == "batch":
        outs, _ = run_batch(s["scans"], precision=PREC[case["precision"]])
        return {k: [_point_parts(o)[k] for o in outs] for k in ("tip", "force", "energy", "steps", "status")}
    if kind == "slab":
        prec = PREC[case["precision"]]
        if case["fresh"]:
            scan = Scan(s["desc"], device=0)
            pts, _ = scan.run(prec)
            scan.close()
            return _point_parts(pts)
        _abi.check(_abi.lib().mafm_scan_build_grid(s["scan"].handle, prec, None))
        s["scan"].run_device(s["out"].data_ptr(), prec)
        return _point_parts(s["out"])
    if kind == "fit":
        fz = fz_image(s["desc"], *s["theta"], precision=PREC[case["precision"]])
        loss = ((fz - s["target"]) ** 2).mean()
        g = torch.autograd.grad(loss, s["theta"])
        return {"fz": fz.detach(), "loss": loss.detach(), "dpos": g[0], "dcharge": g[1], "dpair": g[2]}
    pts, _, _ = s["scan"].run()
    return _point_parts(pts)


# ---- the work of a pass -------------------------------------------------------

# Force evaluations per relaxed point (FIRE, midpoint, tolerances of the
# workloads): measured means of the workloads' scans.
EVALS = {"graphene": 230, "cluster": 157, "slab": 150, "flex": 4000}
# Flops of a tip-atom term: LJ 25, Coulomb 20.
LJ, COUL = 25, 20


def work(case):
    kind = case["kind"]
    if kind == "df_image":
        nw = len(df.weights(case["dz"])[0])
        n, shifts = case["nx"] * case["ny"], case["nz"] - len(df.weights(case["dz"])[0])
        return {"bytes": 16.0 * n * (case["nz"] + shifts), "flops": 4.0 * n * shifts * nw}
    if kind == "flex":
        pts = case["px"] ** 2 * case["nz"]
        return {"bytes": 64.0 * pts, "flops": pts * EVALS["flex"] * 20.0 * (LJ + COUL + 120)}
    if kind == "batch":
        pts = case["scans"] * (case["small"] ** 2 + case["large"] ** 2) / 2 * case["nz"]
        return {"bytes": 64.0 * pts, "flops": pts * EVALS["cluster"] * 127.0 * (LJ + COUL)}
    if kind == "slab":
        n = 2 * (case["px"] - 1) + 31
        nodes = n * n * (2 * (case["nz"] - 1) + 61.0)
        pts = case["px"] ** 2 * case["nz"]
        return {"bytes": nodes * 16 + pts * 64, "flops": nodes * 2048 * 9 * LJ + pts * EVALS["slab"] * 60.0}
    pts = (case["columns"] if kind == "columns" else case["px"] ** 2) * case["nz"]
    atoms = 72 if case.get("system") == "graphene" else case["atoms"]
    per = LJ if case.get("system") == "graphene" else LJ + COUL
    flops = pts * EVALS["graphene" if case.get("system") == "graphene" else "cluster"] * atoms * per
    if kind == "fit":
        flops += pts * atoms * 120.0
    return {"bytes": 64.0 * pts, "flops": float(flops)}


# ---- the same results in 64 bits ------------------------------------------------

class _Relax:
    """FIRE relaxation of every column at once in FP64 torch, from a scan's
    description (rigid pair terms, open boundaries)."""

    def __init__(self, d, theta=None):
        c = d.c
        a = d.atoms()
        f = lambda v: torch.tensor(np.asarray(v), dtype=torch.float64, device="cuda")  # noqa: E731
        self.c = c
        pos, q, pair = theta if theta is not None else (f(a["pos"]), f(a["charge"]), f(d.pair_params()))
        self.pos, self.q, self.pair = pos, q, pair
        t = torch.tensor(a["type"], device="cuda", dtype=torch.long)
        self.type = t
        morse = torch.tensor(d.pair_kinds(), device="cuda", dtype=torch.long)[t] == _abi.PAIR_MORSE
        self.lj_at = torch.nonzero(~morse)[:, 0]
        self.mo_at = torch.nonzero(morse)[:, 0]
        self.coulomb = bool(c.coulomb) and c.tip_charge != 0
        self.k = c.qbase * c.tip_charge

    def s_of(self, x, what):
        """Per-term force factor s (f = s (tip - atom)) and energy of LJ / Morse / Coulomb terms at tips x."""
        at = self.lj_at if what == "lj" else self.mo_at if what == "morse" else None
        pos = self.pos if at is None else self.pos[at]
        dx, dy, dz = (x[:, m:m + 1] - pos[:, m] for m in range(3))
        r2 = dx * dx + dy * dy + dz * dz
        if what == "lj":
            p = self.pair[self.type[at]]
            i2 = 1 / r2
            i6 = i2 * i2 * i2
            tb = p[:, 0] * i6
            ta = p[:, 1] * i6 * i6
            return pos, (12 * ta - 6 * tb) * i2, ta - tb
        r = r2.sqrt()
        if what == "morse":
            p = self.pair[self.type[at]]
            g = torch.exp(-p[:, 1] * (r - p[:, 2]))
            return pos, 2 * p[:, 0] * p[:, 1] * (g * g - g) / r, p[:, 0] * (g * g - 2 * g + 1)
        e = self.k * self.q / r
        return pos, e / r2, e

    def ts(self, x):
        F, E = 0, 0
        kinds = (["lj"] if len(self.lj_at) else []) + (["morse"] if len(self.mo_at) else [])
        for what in kinds + (["coul"] if self.coulomb else []):
            pos, s, e = self.s_of(x, what)
            F = F + (x * s.sum(1, keepdim=True) - s @ pos)
            E = E + e.sum(1)
        return F, E

    def td(self, x, dum):
        c = self.c
        p = c.dummy_pair.p
        r = dum - x
        r2 = (r * r).sum(1, keepdim=True)
        if c.dummy_pair.kind == _abi.PAIR_MORSE:
            rl = r2.sqrt()
            g = torch.exp(-p[1] * (rl - p[2]))
            s, e = 2 * p[0] * p[1] * (g * g - g) / rl, p[0] * (g * g - 2 * g + 1)
        else:
            i2 = 1 / r2
            i6 = i2 * i2 * i2
            s, e = (12 * p[1] * i6 * i6 - 6 * p[0] * i6) * i2, p[1] * i6 * i6 - p[0] * i6
        if c.tip_dummy_coulomb and c.dummy_charge != 0 and c.tip_charge != 0:
            qq = c.qbase * c.dummy_charge * c.tip_charge
            s, e = s + qq * r2 ** -1.5, e + qq * r2 ** -0.5
        F, E = -s * r, e[:, 0]
        rr = (r[:, 0] ** 2 + r[:, 1] ** 2).sqrt()
        dr = rr - c.harm_r0
        E = E + c.harm_k * dr * dr
        k = torch.where(rr > 1e-10, 2 * c.harm_k * dr / rr.clamp_min(1e-300), torch.zeros_like(rr))
        lateral = torch.stack([k * r[:, 0], k * r[:, 1], torch.zeros_like(k)], 1)
        return F + lateral, E

    def step(self, x, v, dum, dt):
        """One integrator step: new positions, velocities, and the step's force and energy."""
        def force(y):
            F, E = self.ts(y)
            f, e = self.td(y, dum)
            return F + f, E + e
        h = dt / 2
        if self.c.integrator == 0:
            F, E = force(x)
            return x + dt * v, v + dt * F, F, E
        f1, e1 = force(x)
        p2, v2 = x + h * v, v + h * f1
        f2, e2 = force(p2)
        if self.c.integrator == 1:
            return x + dt * v2, v + dt * f2, f2, e2
        p3, v3 = x + h * v2, v + h * f2
        f3, e3 = force(p3)
        p4, v4 = x + dt * v3, v + dt * f3
        f4, e4 = force(p4)
        six = dt / 6
        return (x + six * (v + 2 * v2 + 2 * v3 + v4), v + six * (f1 + 2 * f2 + 2 * f3 + f4),
                (f1 + 2 * f2 + 2 * f3 + f4) / 6, (e1 + 2 * e2 + 2 * e3 + e4) / 6)

    def height(self, X, V, En, dum):
        """FIRE at one height for all columns; X, V, En in place; returns the step counts."""
        c = self.c
        n = len(X)
        N = torch.full((n,), c.maxsteps, dtype=torch.int32, device="cuda")
        idx = torch.arange(n, device="cuda")
        x, v, en, d = X.clone(), V.clone(), En.clone(), dum
        dt = torch.full((n, 1), c.dt, dtype=torch.float64, device="cuda")
        al = torch.full((n, 1), 0.1, dtype=torch.float64, device="cuda")
        nn = torch.zeros((n, 1), dtype=torch.int32, device="cuda")
        run = torch.ones(n, dtype=torch.bool, device="cuda")
        for it in range(1, c.maxsteps):
            x1, w, F, E = self.step(x, v, d, dt)
            fl = F.norm(dim=1, keepdim=True)
            e_ok, f_ok = (E - en).abs() < c.etol, fl[:, 0] < c.ftol
            conv = e_ok if c.minterm == 0 else f_ok if c.minterm == 1 else e_ok & f_ok
            m = run[:, None]
            x, en = torch.where(m, x1, x), torch.where(run, E, en)
            N[idx[run & conv]] = it
            pw = (w * F).sum(1, keepdim=True)
            mixed = (1 - al) * w + al * torch.where(fl > 1e-10, F / fl, torch.zeros_like(F)) * w.norm(dim=1, keepdim=True)
            neg = pw < 0
            fast = ~neg & (nn > 5)
            new_v = torch.where(conv[:, None], w, torch.where(neg, torch.zeros_like(w), mixed))
            v = torch.where(m, new_v, v)
            dt = torch.where(neg, dt * 0.5, torch.where(fast, (dt * 1.1).clamp_max(10 * c.dt), dt))
            al = torch.where(neg, torch.full_like(al, 0.1), torch.where(fast, al * 0.99, al))
            nn = torch.where(neg, torch.zeros_like(nn), nn + 1)
            run = run & ~conv
            if it % 8 == 0 or it == c.maxsteps - 1:
                X[idx], V[idx], En[idx] = x, v, en
                keep = torch.nonzero(run)[:, 0]
                if len(keep) == 0:
                    break
                if len(keep) < 0.8 * len(idx):
                    idx, x, v, en, d = idx[keep], x[keep], v[keep], en[keep], d[keep]
                    dt, al, nn, run = dt[keep], al[keep], nn[keep], run[keep]
        return N

    def columns(self, cols):
        """Points (n_cols * nz records) of the listed columns: tip, force, energy, steps, status."""
        c = self.c
        cols = torch.as_tensor(np.asarray(cols), device="cuda", dtype=torch.long)
        n = len(cols)
        i, j = torch.div(cols, c.ny, rounding_mode="floor").double(), (cols % c.ny).double()
        dum = torch.stack([i * c.dx, j * c.dy, torch.full_like(i, c.zhigh)], 1)
        X = dum.clone()
        X[:, 2] = c.zhigh - c.tip_dummy_d
        V, En = torch.zeros_like(X), torch.zeros(n, dtype=torch.float64, device="cuda")
        out = {k: [] for k in ("tip", "force", "energy", "steps", "status")}
        for _ in range(c.nz):
            N = self.height(X, V, En, dum)
            F, E = self.ts(X)
            out["tip"].append(X.clone())
            out["force"].append(F)
            out["energy"].append(E)
            out["steps"].append(N)
            out["status"].append((N >= c.maxsteps).int())
            dum = dum.clone()
            dum[:, 2] -= c.dz
            X[:, 2] -= c.dz
        return {k: torch.stack(v, 1).reshape((n * c.nz,) + v[0].shape[1:]) for k, v in out.items()}

    def gradients(self, x, dum, w):
        """sum_p mu_p . dF_ts(x_p)/dtheta with mu = w (e_z - J^-T dF_ts,z/dx) at the relaxed tips x."""
        n = len(x)
        mu = torch.empty_like(x)
        chunk = 65536
        for b in range(0, n, chunk):
            y = x[b:b + chunk].clone().requires_grad_(True)
            dd = dum[b:b + chunk]
            F = self.ts(y)[0]
            T = self.td(y, dd)[0]
            rows = lambda A: torch.stack([torch.autograd.grad(A[:, m].sum(), y, retain_graph=True)[0]  # noqa: E731
                                          for m in range(3)], 1)
            Jts = rows(F)
            r = torch.hypot(y[:, 0] - dd[:, 0], y[:, 1] - dd[:, 1])
            Jtd = torch.nan_to_num(rows(T))
            if self.c.harm_r0 == 0.0:   # the spring's derivative at the axis
                on = (r <= 1e-10)[:, None, None]
                flat = torch.zeros_like(Jtd)
                flat[:, 0, 0] = flat[:, 1, 1] = -2 * self.c.harm_k
                Jtd = torch.where(on, Jtd + flat, Jtd)
            J = (Jts + Jtd).detach()
            lam = torch.linalg.solve(J.transpose(1, 2), Jts[:, 2].detach()[:, :, None])[:, :, 0]
            ez = torch.zeros_like(lam)
            ez[:, 2] = 1
            mu[b:b + chunk] = w[b:b + chunk, None] * (ez - lam)
        theta = [t.clone().requires_grad_(True) for t in (self.pos, self.q, self.pair)]
        keep = (self.pos, self.q, self.pair)
        self.pos, self.q, self.pair = theta
        tot = [torch.zeros_like(t) for t in theta]
        for b in range(0, n, chunk):
            F = self.ts(x[b:b + chunk])[0]
            g = torch.autograd.grad((mu[b:b + chunk] * F).sum(), theta, allow_unused=True)
            tot = [a if q is None else a + q for a, q in zip(tot, g)]
        self.pos, self.q, self.pair = keep
        return tot


def exact(case, seed):
    kind = case["kind"]
    if kind == "df_image":
        fz = _fz_stack(case, seed).cpu().numpy()
        w, fac = _giessibl(case["dz"])
        nz, nw = case["nz"], len(w)
        g = torch.Generator(device="cuda").manual_seed(seed + 7)
        grad = torch.randn(nz - nw, case["nx"], case["ny"], generator=g, device="cuda", dtype=torch.float64)
        grad = grad.cpu().numpy()
        up = fz[:, :, ::-1]                                  # ascending heights
        img = np.zeros((nz - nw, case["nx"], case["ny"]))
        back = np.zeros_like(up)
        for s in range(nz - nw):
            img[s] = -fac * case["dz"] * (up[:, :, s:s + nw] @ w)
            back[:, :, s:s + nw] += -fac * case["dz"] * grad[s][:, :, None] * w
        return {"df": img, "dfz": np.ascontiguousarray(back[:, :, ::-1])}
    if kind not in ("run", "columns", "fit"):
        return None   # a batch, a 2048-atom periodic grid, a flexible molecule: minutes in torch
    if kind == "run" and (case["px"] ** 2 * case["nz"] > 450_000 or case["integrator"] == "rk4"):
        return None
    if kind == "run" and case["precision"] == "fp32c":
        return None   # its rounding flips steps of the minimiser: points differ by those, not by its precision
    if kind == "fit":
        if case["precision"] == "fp32c" or case["px"] ** 2 * case["nz"] * case["atoms"] > 41_000_000:
            return None
        desc = _load(_scan_spec(dict(case, system="cluster", step=0.1), seed)).desc()
    else:
        desc = _load(_scan_spec(case, seed)).desc()
    rel = _Relax(desc)
    if kind == "columns":
        rng = np.random.default_rng(seed)
        return rel.columns(np.sort(rng.choice(desc.n_columns, case["columns"], replace=False)))
    with torch.no_grad():
        pts = rel.columns(np.arange(desc.n_columns))
    if kind == "run":
        return pts
    c = desc.c
    fz = pts["force"][:, 2].reshape(desc.shape)
    target = _target(case, seed).cuda()
    loss = ((fz - target) ** 2).mean()
    w = (2 * (fz - target) / fz.numel()).reshape(-1)
    i = torch.arange(c.nx, device="cuda", dtype=torch.float64)[:, None, None] * c.dx
    j = torch.arange(c.ny, device="cuda", dtype=torch.float64)[None, :, None] * c.dy
    k = c.zhigh - torch.arange(c.nz, device="cuda", dtype=torch.float64)[None, None, :] * c.dz
    dum = torch.stack([t.expand(desc.shape) for t in (i, j, k)], 3).reshape(-1, 3)
    dpos, dq, dpair = rel.gradients(pts["tip"], dum, w)
    return {"fz": fz, "loss": loss, "dpos": dpos, "dcharge": dq, "dpair": dpair}


def _giessibl(dz, amplitude=0.5, k=1800 * 1.438978, f0=25.0e3):
    """Window weights and prefactor of the frequency-shift sum."""
    fac = (f0 / (2 * k)) * (2 / (np.pi * amplitude * amplitude))
    if (1 + amplitude / dz) % (1 + amplitude // dz) < 0.01:
        amplitude += dz / 2
    z = np.arange(0.0, amplitude + dz, dz)
    z = np.concatenate([-z[:1:-1], z])[1:-1]
    return z / np.sqrt(np.abs(amplitude ** 2 - z ** 2)), fac
