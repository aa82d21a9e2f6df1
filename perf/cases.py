"""The work a user of topopt_gb300 has it do, as cases whose time can be measured.

Kinds of case, each one public call (or the calls of one step) on host data, as
the reference's callers make them:

  compliance   simp_compliance: one certification-style solve with its
               sensitivities, everything built and dropped within the call
  analyze      analyze_fixed_design: the same solve, then the stress field
  optimize     simp_optimize: a short run from the uniform start (OC, MMA, the
               Heaviside-projected update, or the masked overload)
  step         one design iteration of a resident SimpJob whose design arrives
               from and returns to page-locked host memory
  serve        a batch of seeded designs through the serving loop
  homogenize   C^H of a batch of periodic unit cells, all six strains

Every system is solved to 1e-10, the tolerance of this repository's parity
tests: the forms and schedules agree there, so outputs can be compared.
Densities are smooth seeded fields squeezed between 0.02 and 1, what a run's
designs look like after a few iterations; loads are seeded.
"""
import math

import numpy as np
import torch

import topopt_gb300 as tg
from topopt_gb300 import lattice, workloads

TOL = 1e-10
PREC = {"fp64": tg.PREC_FP64, "mixed": tg.PREC_MIXED}
PENALTY, RHO_MIN, NU, MOVE = 3.0, 1e-3, 0.3, 0.2


def _grid(name, kind, nx, ny, nz, precision, **more):
    case = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": precision,
            "radius": 1.5, "volfrac": 0.4}
    case.update(more)
    if name:
        case = dict(name=name, **case)
    return case


def listed():
    return [
        # The smallest call there is: the cantilever of the smoke check, in the
        # default form.  Launches and waits are all it costs.
        _grid("compliance_24x8x8_fp64", "compliance", 24, 8, 8, "fp64"),
        # The projected continuation on the clamped-beam benchmark's grid.
        _grid("projected_48x8x8_fp64", "optimize", 48, 8, 8, "fp64", updater="projected",
              iterations=6, volfrac=0.3),
        # The 60x20x20 cantilever of the golden runs, started afresh.
        _grid("optimize_60x20x20_mixed", "optimize", 60, 20, 20, "mixed", updater="oc",
              iterations=8, volfrac=0.3),
        # A part with empty pockets, frozen regions and odd extents.
        _grid("masked_57x31x23_mixed", "optimize", 57, 31, 23, "mixed", updater="masked",
              iterations=4, radius=2.0),
        # Certifying a part in the default form, extents that turn odd as they halve.
        _grid("compliance_60x36x28_fp64", "compliance", 60, 36, 28, "fp64"),
        # One iteration of a resident job in the default form.
        _grid("step_96x48x48_fp64", "step", 96, 48, 48, "fp64"),
        # The stress analysis that ends a run, extents with odd halves.
        _grid("analyze_108x62x28_mixed", "analyze", 108, 62, 28, "mixed"),
        # One iteration of a mid-size job in the throughput form.
        _grid("step_128x64x64_mixed", "step", 128, 64, 64, "mixed"),
        # The headline design iteration: 4.2 M elements resident.
        _grid("step_256x128x128_mixed", "step", 256, 128, 128, "mixed"),
        # The batched workload's designs, eight in flight together.
        {"name": "serve_8_designs_mixed", "kind": "serve", "precision": "mixed", "count": 8,
         "iterations": 3, "sizes": 1},
        # Small unit cells in the default form.
        {"name": "homogenize_8x20_fp64", "kind": "homogenize", "precision": "fp64", "count": 8,
         "vpc": 20},
        # A sweep of the homogenization workload's 32^3 gyroid and octet cells.
        {"name": "homogenize_32x32_mixed", "kind": "homogenize", "precision": "mixed", "count": 32,
         "vpc": 32},
    ]


def _dims(rng, lo, hi):
    """Extents of a box of about lo .. hi elements (its logarithm uniform), odd
    and even ones, at the aspects of the listed grids."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    ay, az = rng.uniform(0.3, 0.6), rng.uniform(0.3, 0.6)
    nx = (n / (ay * az)) ** (1.0 / 3.0)
    dims = [max(8, round(nx)), max(6, round(ay * nx)), max(6, round(az * nx))]
    if rng.random() < 0.6:  # as most callers: extents that halve a few times
        dims = [max(8, 8 * round(v / 8)) for v in dims]
    return dims


def draw(rng):
    kind = rng.choice(["compliance", "analyze", "optimize", "optimize", "step", "step", "step",
                       "serve", "homogenize", "homogenize"])
    precision = rng.choice(["fp64", "mixed", "mixed"])
    if kind == "serve":
        return {"kind": kind, "precision": "mixed", "count": rng.randint(2, 8),
                "iterations": rng.randint(2, 3), "sizes": rng.randrange(1 << 30)}
    if kind == "homogenize":
        vpc = rng.choice([8, 12, 16, 20, 24, 27, 32])
        most = 8 if precision == "fp64" else 32
        return {"kind": kind, "precision": precision, "vpc": vpc,
                "count": max(1, round(math.exp(rng.uniform(0.0, math.log(most)))))}
    # Odd extents cost the default form's padded coarsening many iterations, so
    # its grids stay below the mixed form's.
    most = {"compliance": 300000, "analyze": 300000, "optimize": 120000, "step": 3000000}[kind]
    nx, ny, nz = _dims(rng, 1500, most if precision == "mixed" else min(most, 220000))
    if precision == "fp64":
        nx, ny, nz = (max(8, 8 * round(v / 8)) for v in (nx, ny, nz))
    case = _grid(None, kind, nx, ny, nz, precision, radius=round(rng.uniform(1.2, 2.5), 2),
                 volfrac=round(rng.uniform(0.25, 0.5), 2))
    if kind == "optimize":
        case["updater"] = rng.choice(["oc", "oc", "mma", "projected", "masked"])
        case["iterations"] = rng.randint(2, 5)
    return case


# ------------------------------------------------------------------- inputs
def _field(case, seed):
    """A smooth seeded density of mean about volfrac in [0.02, 1]."""
    rng = np.random.default_rng(seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = 0.0
    for _ in range(10):
        t = []
        for n in (case["nz"], case["ny"], case["nx"]):
            k, ph = rng.integers(1, 5), rng.uniform(0.0, 2.0 * np.pi)
            t.append(torch.from_numpy(np.cos(np.pi * k * np.linspace(0.0, 1.0, n) + ph)).to(dev))
        f = f + rng.normal() * torch.einsum("i,j,k->ijk", *t)
    f = (f - f.mean()) / f.std()
    lo, hi = -6.0, 6.0
    for _ in range(30):
        mid = 0.5 * (lo + hi)
        r = 0.02 + 0.98 * torch.sigmoid(2.5 * (f - mid))
        lo, hi = (mid, hi) if float(r.mean()) > case["volfrac"] else (lo, mid)
    return r.reshape(-1).cpu().numpy()


def _tags_and_mask(case, seed):
    """A masked part: an empty pocket, a frozen-solid pad and a frozen-void hole,
    all away from the clamped and the loaded face."""
    rng = np.random.default_rng(seed + 7)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    tags = np.ones((nz, ny, nx), np.uint8)
    mask = np.full((nz, ny, nx), tg.MASK_ACTIVE, np.uint8)
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")

    def ball(where, r):
        c = [rng.uniform(0.3, 0.7) * n for n in (nz, ny)] + [where * nx]
        return (z - c[0]) ** 2 + (y - c[1]) ** 2 + (x - c[2]) ** 2 < (r * min(ny, nz)) ** 2

    tags[ball(rng.uniform(0.25, 0.35), 0.2)] = 0
    mask[ball(rng.uniform(0.45, 0.55), 0.2)] = tg.MASK_FROZEN_SOLID
    mask[ball(rng.uniform(0.65, 0.75), 0.2)] = tg.MASK_FROZEN_VOID
    return tags.ravel(), mask.ravel()


def _problem(case, seed):
    tags = mask = None
    if case.get("updater") == "masked":
        tags, mask = _tags_and_mask(case, seed)
    bcs, loads = workloads.cantilever_seeded_load(case["nx"], case["ny"], case["nz"], seed)
    return tg.Problem(case["nx"], case["ny"], case["nz"], 1.0, tags, bcs, loads), mask


def _options(case):
    o = tg.SimpOptions(volume_fraction=case["volfrac"], filter_radius=case["radius"], move=MOVE,
                       change_tol=0.0, cg_tolerance=TOL,
                       max_iterations=case.get("iterations", 1),
                       solve=tg.SolveOptions(precision=PREC[case["precision"]]))
    if case.get("updater") == "mma":
        o.updater = tg.UPDATER_MMA
    if case.get("updater") == "projected":
        half = case["iterations"] // 2
        o.projection = [(1.0, 0.2, half), (2.0, 0.2, case["iterations"] - half)]
    return o


def _cells(case, seed):
    return lattice.batch(case["count"], case["vpc"], seed)[0]


def _designs(case, seed):
    """The workload's seeded designs at its range of extents (32 .. 128 x 16 .. 64
    x 16 .. 64, even), which belong to the case: "sizes" seeds them."""
    sizes, rng = np.random.default_rng(case["sizes"]), np.random.default_rng(seed)
    made = []
    for _ in range(case["count"]):
        dims = [2 * int(sizes.integers(lo, hi)) for lo, hi in ((16, 65), (8, 33), (8, 33))]
        pb, params, opt = workloads.design(int(rng.integers(1 << 31)), PREC[case["precision"]],
                                           case["iterations"], dims)
        opt.cg_tolerance = TOL
        made.append((pb, params, opt))
    return made


def prepare(case, seed):
    kind = case["kind"]
    if kind == "homogenize":
        return {"case": case, "cells": _cells(case, seed)}
    if kind == "serve":
        return {"case": case, "designs": _designs(case, seed),
                "server": tg.Server(64 << 30, max_active=8)}
    pb, mask = _problem(case, seed)
    state = {"case": case, "pb": pb, "mask": mask, "params": tg.SimpParams(),
             "options": _options(case)}
    if kind in ("compliance", "analyze"):
        state["rho"] = _field(case, seed)
    if kind == "step":
        state["job"] = tg.SimpJob(pb, state["params"], state["options"])
        for name in ("in", "x", "xphys"):
            state[name] = tg.host_array(pb.nv)
        state["in"][:] = _field(case, seed)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "compliance":
        r = tg.simp_compliance(state["pb"], state["params"], state["rho"], tolerance=TOL,
                               options=state["options"].solve)
        return {"u": r["u"], "dcompliance": r["dcompliance"], "compliance": r["compliance"]}
    if kind == "analyze":
        r = tg.analyze_fixed_design(state["pb"], state["params"], state["rho"], tg.StrengthSpec(),
                                    cg_tolerance=TOL, solve=state["options"].solve, fields=True)
        return {k: r[k] for k in ("von_mises", "stress", "displacement", "compliance",
                                  "max_von_mises", "max_interlayer_tension", "printed_voxels")}
    if kind == "optimize":
        r = tg.simp_optimize(state["pb"], state["params"], state["options"], mask=state["mask"])
        return {"design": r["design"], "physical_density": r["physical_density"],
                "compliance": np.array([h["compliance"] for h in r["history"]])}
    if kind == "step":
        job = state["job"]
        job.write_design(state["in"])
        row = job.step()
        job.read(state["x"], state["xphys"])
        return {"design": state["x"], "physical_density": state["xphys"],
                "compliance": row["compliance"], "change": row["change"],
                "volume_fraction": row["volume_fraction"]}
    if kind == "serve":
        tickets = [state["server"].submit(*d) for d in state["designs"]]
        out = [state["server"].wait(t) for t in tickets]
        return [{"design": r["design"], "physical_density": r["physical_density"],
                 "compliance": r["compliance"]} for r in out]
    return tg.homogenize(state["cells"], tolerance=TOL, precision=PREC[case["precision"]])[0]


# --------------------------------------------------------------------- work
def work(case):
    """Bytes: every host input and output once.  Flops: the reference's own count
    of 1152 per element and operator apply, for the applies that solving these
    systems to the tolerance cannot do without at the multigrid's best rate
    (about 20 iterations of 3 applies; 100 of one apply for the unpreconditioned
    periodic systems, per strain)."""
    if case["kind"] == "homogenize":
        nv = case["count"] * case["vpc"] ** 3
        return {"bytes": nv + 288.0 * case["count"], "flops": nv * 6 * 100 * 1152.0}
    if case["kind"] == "serve":  # the designs' mean size
        nv = case["count"] * 80 * 40 * 40
        return {"bytes": 16.0 * nv, "flops": nv * case["iterations"] * 60 * 1152.0}
    nv = case["nx"] * case["ny"] * case["nz"]
    ndof = 3 * (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    io = {"compliance": 16 * nv + 8 * ndof, "analyze": 64 * nv + 8 * ndof, "optimize": 16 * nv,
          "step": 24 * nv}[case["kind"]]
    return {"bytes": float(io), "flops": case.get("iterations", 1) * nv * 60 * 1152.0}


# -------------------------------------------- the same in plain 64-bit torch
_CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0),
            (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def _elastic():
    d = np.zeros((6, 6))
    c = 1.0 / ((1.0 + NU) * (1.0 - 2.0 * NU))
    d[:3, :3] = c * NU
    d[range(3), range(3)] = c * (1.0 - NU)
    d[range(3, 6), range(3, 6)] = c * (1.0 - 2.0 * NU) / 2.0
    return d


def _strain_matrix(p):
    """Strains [xx, yy, zz, xy, yz, zx] of the unit hex at p in [-1, 1]^3."""
    b = np.zeros((6, 24))
    for a, o in enumerate(_CORNERS):
        s = [2 * v - 1 for v in o]
        f = [1.0 + s[i] * p[i] for i in range(3)]
        gx, gy, gz = (0.25 * s[0] * f[1] * f[2], 0.25 * s[1] * f[0] * f[2],
                      0.25 * s[2] * f[0] * f[1])
        b[0, 3 * a], b[1, 3 * a + 1], b[2, 3 * a + 2] = gx, gy, gz
        b[3, 3 * a], b[3, 3 * a + 1] = gy, gx
        b[4, 3 * a + 1], b[4, 3 * a + 2] = gz, gy
        b[5, 3 * a], b[5, 3 * a + 2] = gz, gx
    return b


def _stiffness():
    g = 1.0 / math.sqrt(3.0)
    k = np.zeros((24, 24))
    for p in [(x, y, z) for x in (-g, g) for y in (-g, g) for z in (-g, g)]:
        b = _strain_matrix(p)
        k += b.T @ _elastic() @ b / 8.0
    return k


def _dev(a):
    return torch.as_tensor(a, dtype=torch.float64, device="cuda" if torch.cuda.is_available()
                           else "cpu")


class _Elasticity:
    """K u on a voxel grid with element moduli E (nz, ny, nx), or on the torus;
    u has the shape (..., 3, z, y, x)."""

    def __init__(self, E, periodic):
        self.E, self.periodic, self.ke = E, periodic, _dev(_stiffness())

    def corners(self, u):
        nz, ny, nx = self.E.shape
        if self.periodic:
            v = [torch.roll(u, (-o[2], -o[1], -o[0]), (-3, -2, -1)) for o in _CORNERS]
        else:
            v = [u[..., o[2]:o[2] + nz, o[1]:o[1] + ny, o[0]:o[0] + nx] for o in _CORNERS]
        return torch.stack(v, -5).flatten(-5, -4)  # (..., 24, z, y, x)

    def gather(self, f, like):
        nz, ny, nx = self.E.shape
        out = torch.zeros_like(like)
        for a, o in enumerate(_CORNERS):
            fa = f[..., 3 * a:3 * a + 3, :, :, :]
            if self.periodic:
                out += torch.roll(fa, (o[2], o[1], o[0]), (-3, -2, -1))
            else:
                out[..., o[2]:o[2] + nz, o[1]:o[1] + ny, o[0]:o[0] + nx] += fa
        return out

    def forces(self, u):
        return torch.einsum("ij,...jzyx->...izyx", self.ke, self.corners(u))

    def apply(self, u):
        return self.gather(self.E * self.forces(u), u)

    def diagonal(self, like):
        d = torch.diagonal(self.ke).reshape(24, 1, 1, 1) * self.E
        return self.gather(d.expand(*like.shape[:-4], *d.shape), like)

    def solve(self, b, free, tol=1e-13, most=20000):
        """Jacobi-preconditioned CG on the free DOFs, all leading systems together."""
        b = b * free
        dims = (-4, -3, -2, -1)
        d = self.diagonal(b)
        inv = torch.where((d > 0) & (free > 0), 1.0 / torch.where(d > 0, d, 1.0), 0.0)
        x, r = torch.zeros_like(b), b.clone()
        z = inv * r
        p, rz = z.clone(), (r * z).sum(dims, keepdim=True)
        b2 = (b * b).sum(dims, keepdim=True)
        for k in range(most):
            ap = self.apply(p) * free
            pap = (p * ap).sum(dims, keepdim=True)
            alpha = torch.where(pap > 0, rz / torch.where(pap > 0, pap, 1.0), 0.0)
            x += alpha * p
            r -= alpha * ap
            if k % 16 == 15 and bool(((r * r).sum(dims, keepdim=True) <= tol * tol * b2).all()):
                break
            z = inv * r
            new = (r * z).sum(dims, keepdim=True)
            p = z + torch.where(rz > 0, new / torch.where(rz > 0, rz, 1.0), 0.0) * p
            rz = new
        return x


class _Simp:
    """The reference's SIMP pieces on (nz, ny, nx) fields."""

    def __init__(self, case, seed):
        pb, mask = _problem(case, seed)
        self.case, self.shape = case, (pb.nz, pb.ny, pb.nx)
        solid = np.ones(pb.nv, bool) if pb.tags is None else pb.tags != 0
        pins = np.where(solid, tg.MASK_ACTIVE if mask is None else mask, tg.MASK_FROZEN_VOID)
        self.design = _dev(solid if mask is None else pins == tg.MASK_ACTIVE).reshape(self.shape)
        self.elem = _dev(solid if mask is None else pins != tg.MASK_FROZEN_VOID).reshape(self.shape)
        self.pins = None if mask is None else _dev(pins).reshape(self.shape)
        node = (3, pb.nz + 1, pb.ny + 1, pb.nx + 1)

        def vector(entries, default):
            v = np.full((pb.nnodes, 3), default)
            for n, c, value in entries:
                v[n, c] = value if default == 0.0 else 0.0
            return _dev(np.ascontiguousarray(v.T)).reshape(node)

        self.load, self.free = vector(pb.loads, 0.0), vector(pb.bcs, 1.0)
        r = case["radius"]
        m = int(math.floor(r))
        self.taps = [(dz, dy, dx, r - math.sqrt(dx * dx + dy * dy + dz * dz))
                     for dz in range(-m, m + 1) for dy in range(-m, m + 1)
                     for dx in range(-m, m + 1) if r > math.sqrt(dx * dx + dy * dy + dz * dz)]
        self.m = m
        self.hs = self._conv(self.design) * self.design
        self.dv = self.adjoint(self.design)

    def _conv(self, v):
        m, (nz, ny, nx) = self.m, self.shape
        p = torch.nn.functional.pad(v, [m] * 6)
        return sum(w * p[m + dz:m + dz + nz, m + dy:m + dy + ny, m + dx:m + dx + nx]
                   for dz, dy, dx, w in self.taps)

    def filter(self, x):
        h = self.hs > 0
        return torch.where(h, self._conv(x * self.design) / torch.where(h, self.hs, 1.0), 0.0)

    def adjoint(self, s):
        h = self.hs > 0
        return self._conv(torch.where(h, s / torch.where(h, self.hs, 1.0), 0.0)) * self.design

    def physical(self, x):
        xp = self.filter(x)
        if self.pins is not None:
            xp = torch.where(self.pins == tg.MASK_FROZEN_SOLID, 1.0,
                             torch.where(self.pins == tg.MASK_FROZEN_VOID, 0.0, xp))
        return xp

    def solve(self, rho):
        r = rho.clamp(RHO_MIN, 1.0)
        op = _Elasticity(r ** PENALTY * self.elem, False)
        touched = op.gather(self.elem.expand(24, *self.shape), self.load) > 0
        u = op.solve(self.load, self.free * touched)
        q = (op.corners(u) * op.forces(u)).sum(0)
        c = float((r ** PENALTY * self.elem * q).sum())
        return u, c, -PENALTY * r ** (PENALTY - 1.0) * q * self.elem

    def update(self, x, dc):
        dcf, d = self.adjoint(dc), self.design > 0
        target = self.case["volfrac"] * float(self.design.sum())
        lo, hi = (x - MOVE).clamp(min=RHO_MIN), (x + MOVE).clamp(max=1.0)

        def candidate(lam):
            b = torch.where(self.dv > 0, -dcf / (lam * torch.where(self.dv > 0, self.dv, 1.0)), 0.0)
            t = torch.minimum(torch.maximum(x * b.clamp(min=0.0).sqrt(), lo), hi)
            return torch.where(d, t, x if self.pins is not None else torch.zeros_like(x))

        def exceeds(lam):
            return float((self.filter(candidate(lam)) * self.design).sum()) > target

        l1, l2 = 0.0, 1.0
        while l2 < 1e30 and exceeds(l2):
            l2 *= 2.0
        for _ in range(100):
            if not l2 - l1 > 1e-6 * (l1 + l2):
                break
            mid = 0.5 * (l1 + l2)
            l1, l2 = (mid, l2) if exceeds(mid) else (l1, mid)
        return candidate(0.5 * (l1 + l2))

    def step(self, x):
        _, c, dc = self.solve(self.physical(x))
        new = self.update(x, dc)
        return new, self.physical(new), c

    def nodes(self, u):
        return np.ascontiguousarray(u.reshape(3, -1).T.cpu().numpy()).ravel()


def _exact_cells(case, seed):
    out = []
    ke = _stiffness()
    chi0 = np.zeros((24, 6))
    for a, (ox, oy, oz) in enumerate(_CORNERS):
        chi0[3 * a, 0], chi0[3 * a + 1, 1], chi0[3 * a + 2, 2] = ox, oy, oz
        chi0[3 * a, 3], chi0[3 * a + 1, 4], chi0[3 * a + 2, 5] = oy, oz, ox
    f0 = ke @ chi0
    for cell in _cells(case, seed):
        solid = _dev(cell != 0)
        op = _Elasticity(solid, True)
        fe = _dev(f0.T).reshape(6, 24, 1, 1, 1) * solid
        like = torch.zeros((6, 3) + tuple(solid.shape), dtype=torch.float64, device=solid.device)
        f = op.gather(fe, like)
        free = (op.gather(solid.expand(6, 24, *solid.shape), like) > 0).double()
        free[:, :, 0, 0, 0] = 0.0
        chi = op.solve(f, free)
        c0 = _dev(chi0.T @ f0) * solid.sum()
        out.append((c0 - torch.einsum("iczyx,jczyx->ij", f, chi)) / solid.numel())
    return torch.stack(out).cpu().numpy()


def exact(case, seed):
    if case["kind"] == "homogenize":
        return _exact_cells(case, seed)
    if case["kind"] == "serve" or case.get("updater") in ("mma", "projected"):
        return None
    nv = case["nx"] * case["ny"] * case["nz"]
    if nv * case.get("iterations", 1) > 600000:
        return None  # minutes of unpreconditioned iterations
    s = _Simp(case, seed)
    if case["kind"] == "step":
        x = _dev(_field(case, seed)).reshape(s.shape)
        new, xp, c = s.step(x)
        return {"design": new.reshape(-1), "physical_density": xp.reshape(-1), "compliance": c,
                "change": float((new - x).abs().max()),
                "volume_fraction": float((xp * s.design).sum() / s.design.sum())}
    if case["kind"] == "optimize":
        x = case["volfrac"] * s.design
        if s.pins is not None:
            x = torch.where(s.pins == tg.MASK_FROZEN_SOLID, 1.0, x)
        history = []
        for _ in range(case["iterations"]):
            x, xp, c = s.step(x)
            history.append(c)
        return {"design": x.reshape(-1), "physical_density": xp.reshape(-1),
                "compliance": np.array(history)}
    rho = _dev(_field(case, seed)).reshape(s.shape)
    u, c, dc = s.solve(rho)
    if case["kind"] == "compliance":
        return {"u": s.nodes(u), "dcompliance": dc.reshape(-1), "compliance": c}
    op = _Elasticity(torch.ones(s.shape, dtype=torch.float64, device=rho.device), False)
    printed = (rho > tg.StrengthSpec().printed_iso).double()
    sig = torch.einsum("ij,jzyx->izyx", _dev(_elastic() @ _strain_matrix((0.0, 0.0, 0.0))),
                       op.corners(u)) * printed
    xx, yy, zz, xy, yz, zx = sig
    vm = (0.5 * ((xx - yy) ** 2 + (yy - zz) ** 2 + (zz - xx) ** 2)
          + 3.0 * (xy ** 2 + yz ** 2 + zx ** 2)).sqrt()
    touched = op.gather(printed.expand(24, *s.shape), u) > 0
    return {"von_mises": vm.reshape(-1), "stress": sig.reshape(6, -1).T.contiguous(),
            "displacement": s.nodes(u * touched), "compliance": c,
            "max_von_mises": float(vm.max()), "max_interlayer_tension": None,
            "printed_voxels": int(printed.sum())}
