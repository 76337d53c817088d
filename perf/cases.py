"""The work that a user of this package has it do, as cases that can be timed.

A case names a kind of call and its sizes:

  fields    set the magnetisation, evaluate H_eff and the energies, field after
            field (the precision study of many random states on one mesh)
  advance   nmag.Simulation: start from a seeded state and advance the BDF
            integrator, reading <m> at every record
  product   the dense boundary (BEM) product for many boundary potentials
  gradient  a differentiable RK4 trajectory: forward, and the gradients of a
            loss on <m>(t) for the per-element material and the field pulses
  particles a batch of particles of uneven size: integrator steps for each
  setup     load a mesh (operators, boundary matrix, solver data) and evaluate
            the first field

Meshes are the boxes of the package's own configurations (30 nm cube, 500 x 125
x 3 nm film, the 250 x 100 x 3 nm profiling film) and boxes of other sizes;
permalloy, with the tolerances of the precision study (1e-12) and of the
trajectory comparisons (1e-10).
"""
import itertools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "nmag-src_gb300"))

MU0 = 4e-7 * math.pi
MS, C_EXCH = 0.86, 24.0583053511          # permalloy, simulation units
H_EXT = tuple(v * 1e-3 / MU0 * 1e-6 for v in (-24.6, 4.3, 0.0))   # (-24.6, 4.3, 0) mT
AXIS = (0.0, 0.6, 0.8)
FORM = {"fp64": 0, "fp32": 1, "fp32x2": 2, "bf16x3": 3}


def _box_case(kind, nx, ny, nz, hx, hy, hz, **more):
    return dict({"kind": kind, "nx": nx, "ny": ny, "nz": nz, "hx": hx, "hy": hy, "hz": hz}, **more)


def _cube(kind, **more):
    return _box_case(kind, 10, 10, 10, 3.0, 3.0, 3.0, **more)


def _film(kind, **more):
    return _box_case(kind, 200, 50, 2, 2.5, 2.5, 1.5, **more)


def _film_small(kind, **more):
    return _box_case(kind, 100, 40, 2, 2.5, 2.5, 1.5, **more)


def listed():
    return [
        # a few dozen nodes: what a script's first tries and unit tests run; latency and launches
        _box_case("fields", 4, 3, 2, 2.0, 2.5, 1.5, name="fields_box60", form="fp64", anis=0.0, count=12, rtol=1e-12),
        # the 30 nm cube with a uniaxial easy axis: an ordinary small sample, state after state
        _cube("fields", name="fields_cube", form="fp64", anis=0.12, count=12, rtol=1e-12),
        # the film, one random state after another: the FP64 side of the precision study
        _film("fields", name="fields_film", form="fp64", anis=0.0, count=12, rtol=1e-12),
        # the cube's dynamics from its seeded state (alpha 0.5): many short integrator steps
        _cube("advance", name="advance_cube", form="fp64", cg="fp64", members=1, anchor=0.0, jv="fp64", alpha=0.5,
              materials=1, rtol=1e-10, ps=1.0, records=4),
        # the film's dynamics in the plain FP64 form
        _film("advance", name="advance_film", form="fp64", cg="fp64", members=1, anchor=0.0, jv="fp64", alpha=0.02,
              materials=1, rtol=1e-10, ps=0.2, records=2),
        # eight films at once in the mixed-precision form that the benchmark runs
        _film("advance", name="advance_film_x8", form="fp32x2", cg="fp32", members=8, anchor=1e-2, jv="fp32",
              alpha=0.02, materials=1, rtol=1e-10, ps=0.2, records=2),
        # two materials side by side in a slab, each with its own magnetisation
        _box_case("advance", 40, 12, 4, 2.5, 2.5, 2.0, name="advance_two_materials", form="fp64", cg="fp64",
                  members=1, anchor=0.0, jv="fp64", alpha=0.1, materials=2, rtol=1e-10, ps=0.3, records=3),
        # 128 boundary potentials through the film's matrix on the tensor cores
        _film("product", name="product_film_bf16x3", form="bf16x3", rhs=128),
        # an uneven number of potentials through the compensated product
        _film_small("product", name="product_slab_fp32x2", form="fp32x2", rhs=21),
        # gradients of a pulse optimisation on the cube, Poisson solves tight
        _cube("gradient", name="gradient_cube", form="fp64", cg="fp64", steps=20, ckpt=10, pulses=4, rtol=1e-12),
        # 40 particles of 125 to 9,261 nodes, two integrator steps each
        {"kind": "particles", "name": "particles_40", "count": 40, "lo": 4, "hi": 20, "launches": 2, "rtol": 1e-7},
        # from a mesh to the first field: what every script pays once
        _film_small("setup", name="setup_slab", form="fp64", rtol=1e-12),
    ]


def draw(rng):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def box(most):   # a box of 2 .. `most` nodes, of any aspect
        while True:
            n = [logint(1, 160), logint(1, 60), logint(1, 14)]
            if 12 <= (n[0] + 1) * (n[1] + 1) * (n[2] + 1) <= most:
                break
        h = [round(rng.uniform(1.5, 3.5), 2) for _ in range(3)]
        return n + h

    kind = rng.choice(("fields", "fields", "advance", "advance", "product", "gradient", "particles", "setup"))
    if kind == "fields":
        return _box_case(kind, *box(12000), form=rng.choice(("fp64", "fp64", "fp32x2")),
                         anis=round(rng.choice((0.0, rng.uniform(0.05, 0.5))), 3), count=rng.randint(11, 14),
                         rtol=1e-12)
    if kind == "advance":
        members = rng.choice((1, 1, 1, 3, 8))
        mixed = members > 1
        return _box_case(kind, *box(12000), form="fp32x2" if mixed else "fp64", cg="fp32" if mixed else "fp64",
                         members=members, anchor=1e-2 if mixed else 0.0, jv="fp32" if mixed else "fp64",
                         alpha=rng.choice((0.5, 0.1, 0.02)), materials=1, rtol=1e-10,
                         ps=round(rng.uniform(0.1, 0.3), 3), records=rng.randint(1, 3))
    if kind == "product":
        return _box_case(kind, *box(14000), form=rng.choice(("fp64", "fp32x2", "bf16x3")), rhs=logint(1, 128))
    if kind == "gradient":
        steps = rng.randint(5, 20)
        return _box_case(kind, *box(4000), form="fp64", cg=rng.choice(("fp64", "fp32")), steps=steps,
                         ckpt=rng.randint(3, steps), pulses=rng.randint(1, 5), rtol=1e-12)
    if kind == "particles":
        lo = rng.randint(2, 8)
        return {"kind": kind, "count": logint(5, 40), "lo": lo, "hi": rng.randint(lo + 2, 18),
                "launches": rng.randint(1, 3), "rtol": 1e-7}
    return _box_case(kind, *box(9000), form=rng.choice(("fp64", "fp32x2")), rtol=1e-12)


# ---- inputs ----

def _box(case):
    """Points (N, 3) and simplices (T, 4) of a box of cells, each split into six tetrahedra."""
    n = np.array([case["nx"], case["ny"], case["nz"]])
    h = np.array([case["hx"], case["hy"], case["hz"]])
    k, j, i = np.meshgrid(*(np.arange(m + 1) for m in n[::-1]), indexing="ij")
    points = np.stack([i, j, k], -1).reshape(-1, 3) * h
    k, j, i = np.meshgrid(*(np.arange(m) for m in n[::-1]), indexing="ij")
    corner = np.stack([i, j, k], -1).reshape(-1, 3)
    step = np.array([1, n[0] + 1, (n[0] + 1) * (n[1] + 1)])
    tets = np.empty((len(corner), 6, 4), np.int32)
    for p, axes in enumerate(itertools.permutations(range(3))):
        at = corner.copy()
        tets[:, p, 0] = at @ step
        for s, a in enumerate(axes):
            at[:, a] += 1
            tets[:, p, s + 1] = at @ step
    return points, tets.reshape(-1, 4)


def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def _states(case, n, seed):
    """`count` random states: every node's direction uniform on the sphere."""
    rng = np.random.default_rng(1000 + seed)
    return [_unit(rng.standard_normal((n, 3))) for _ in range(case["count"])]


def _start(n, seed, base=(1.0, 0.25, 0.1)):
    return _unit(np.asarray(base) + 0.01 * np.random.default_rng(seed).standard_normal((n, 3)))


def _potentials(case, nb, seed):
    """Smooth boundary potentials of different wavelengths, as solves give them."""
    rng = np.random.default_rng(seed)
    k = np.arange(nb)
    w = np.geomspace(1e-4, 3e-1, case["rhs"])
    return 100.0 * np.sin(k[None, :] * w[:, None] + rng.uniform(0.0, 6.28, (case["rhs"], 1)))


def _engine(case, members=0, adjoint_cg="fp64"):
    from nmag import _lib
    mt = _lib.Material()
    mt.Ms, mt.exch_coeff, mt.C1, mt.C2, mt.C3 = MS, C_EXCH, -0.221012, -0.00442023, 0.1
    mt.E_coeff_half, mt.E_coeff_ext = -0.540354, -1.08071
    anis = case.get("anis", 0.0)
    if anis:
        mt.K1, mt.anis_coeff = anis, 2.0 * anis / (1.2566370614 * MS)
        for d in range(3):
            mt.axis[d] = AXIS[d]
    op = _lib.Options()
    op.do_demag = 1
    op.nbc_rtol = op.dbc_rtol = case.get("rtol", 1e-12)
    op.nbc_atol = op.dbc_atol = 1e-50
    op.nbc_maxits = op.dbc_maxits = 20000
    op.bem_precision, op.n_members = FORM[case["form"]], members
    op.adjoint_cg_precision = 1 if adjoint_cg == "fp32" else 0
    points, tets = _box(case)
    return _lib.Engine(points, tets, mt, op)


def _simulation(case, seed):
    import nmag
    from nmag import SI, mesh
    points, tets = _box(case)
    mats = [nmag.MagMaterial("Py", Ms=SI(8.6e5, "A/m"), exchange_coupling=SI(1.3e-11, "J/m"),
                             llg_damping=case["alpha"], llg_gamma_G=SI(2.211e5, "m/A s"))]
    regions = np.ones(len(tets), np.int32)
    if case["materials"] == 2:
        mats.append(nmag.MagMaterial("Co", Ms=SI(1.4e6, "A/m"), exchange_coupling=SI(3.0e-11, "J/m"),
                                     llg_damping=case["alpha"], llg_gamma_G=SI(2.211e5, "m/A s"),
                                     anisotropy=nmag.uniaxial_anisotropy(axis=list(AXIS), K1=SI(5e5, "J/m^3"))))
        x = points[tets].mean(1)[:, 0]
        regions = np.where(x < 0.5 * points[:, 0].max(), 1, 2).astype(np.int32)
    tol = case["rtol"]
    sim = nmag.Simulation("case", bem_precision=case["form"], cg_precision=case["cg"], n_members=case["members"],
                          bem_anchor=case["anchor"], jv_precision=case["jv"],
                          ksp_tolerances={"NBC.rtol": tol, "DBC.rtol": tol})
    sim.load_mesh(mesh.Mesh(points, tets, regions), [(m.name, m) for m in mats], unit_length=SI(1e-9, "m"))
    sim.set_H_ext(np.array(H_EXT) * 1e6, SI(1.0, "A/m"))
    B, n = case["members"], sim.engine.N
    m0 = [_start(n, seed + 31 * b) for b in range(B)]
    return {"sim": sim, "m0": np.stack(m0) if B > 1 else m0[0], "mats": [m.name for m in mats]}


def _gradient_inputs(case, n, n_tets, seed):
    rng = np.random.default_rng(seed)
    return {"m0": _start(n, seed).reshape(-1), "Ms": MS * (1.0 + 0.05 * rng.standard_normal(n_tets)),
            "K1": 0.05 * np.abs(rng.standard_normal(n_tets)),
            "pulses": rng.standard_normal((case["pulses"], 3)) * (5e-3 / MU0) * 1e-6}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fields":
        eng = _engine(case)
        eng.set_h_ext(H_EXT)
        return {"case": case, "eng": eng, "m": _states(case, eng.N, seed)}
    if kind == "advance":
        return dict(_simulation(case, seed), case=case)
    if kind == "product":
        eng = _engine(case)
        x = torch.tensor(_potentials(case, eng.nb, seed), dtype=torch.float64, device="cuda")
        return {"case": case, "eng": eng, "x": x, "y": torch.empty_like(x)}
    if kind == "gradient":
        eng = _engine(case, adjoint_cg=case["cg"])
        eng.set_h_ext(H_EXT)
        d = {k: torch.tensor(v, dtype=torch.float64, device="cuda")
             for k, v in _gradient_inputs(case, eng.N, eng.T, seed).items()}
        for k in ("m0", "Ms", "K1", "pulses"):
            d[k].requires_grad_(True)
        return dict(d, case=case, eng=eng)
    if kind == "particles":
        from nmag.batch import ParticleBatch
        rng = np.random.default_rng(seed)
        # sizes spread evenly over the range, so that another seed is the same amount of work
        parts, ms = [], []
        for k in range(case["count"]):
            c = case["lo"] + int(round((case["hi"] - case["lo"]) * k / max(1, case["count"] - 1)))
            points, tets = _box({"nx": c, "ny": c, "nz": c, "hx": 2.0, "hy": 2.0, "hz": 2.0})
            ms_p, k1 = rng.uniform(0.4, 1.7), rng.uniform(0.0, 0.5)
            axis, hdir = _unit(rng.standard_normal(3)), _unit(rng.standard_normal(3))
            parts.append((points, tets, {"Ms": ms_p, "exch_coeff": 26.0 / (1.2566370614 * ms_p), "C1": -0.218911,
                                         "C2": -0.0218911, "C3": 0.1, "K1": k1, "axis": axis,
                                         "anis_coeff": 2.0 * k1 / (1.2566370614 * ms_p), "E_coeff_half": 0.0,
                                         "E_coeff_ext": 0.0}, hdir))
            ms.append(_unit(hdir + 0.05 * rng.standard_normal((len(points), 3))))
        b = ParticleBatch(parts, n_stages=81, h_max=1.0 / MU0 * 1e-6, rtol=case["rtol"], atol=case["rtol"],
                          cg_rtol=1e-10)
        b.set_m(ms)
        return {"case": case, "batch": b}
    points, tets = _box(case)
    return {"case": case, "m": _states({"count": 1}, len(points), seed)[0]}


# ---- one pass ----

def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "fields":
        eng, out = state["eng"], {"H_total": [], "dmdt": [], "energies": []}
        for m in state["m"]:
            eng.set_m(m)
            f = eng.eval_fields()
            out["H_total"].append(f["H_total"])
            out["dmdt"].append(f["dmdt"])
            out["energies"].append(eng.averages(energies=True)[1])
        return out
    if kind == "advance":
        from nmag import SI
        sim, avg = state["sim"], []
        sim.set_m(state["m0"])
        sim.reinitialise(initial_time=0)
        for k in range(case["records"]):
            sim.advance_time(SI(case["ps"] * (k + 1) / case["records"] * 1e-12, "s"))
            avg.append([sim.get_subfield_average_siv("m_" + n if len(state["mats"]) > 1 else "m")
                        for n in state["mats"]])
        return {"m": sim.engine.get_m(), "average": np.array(avg)}
    if kind == "product":
        state["eng"].bem_apply_device(state["x"].data_ptr(), state["y"].data_ptr(), case["rhs"])
        return state["y"]
    if kind == "gradient":
        from nmag import adjoint
        spp = max(1, case["steps"] // case["pulses"])
        mT, hist = adjoint.rk4_trajectory(state["eng"], state["m0"], state["Ms"], state["K1"], state["pulses"], AXIS,
                                          MS, 1.2566370614, 0.1, case["steps"], case["ckpt"], spp)
        loss = adjoint.film_loss(hist)
        g = torch.autograd.grad(loss, [state[k] for k in ("m0", "Ms", "K1", "pulses")])
        return {"m": mT.detach(), "history": hist.detach(), "loss": loss.detach(), "gradients": list(g)}
    if kind == "particles":
        b = state["batch"]
        b.run(case["launches"])
        st = b.state()
        return {"m": np.concatenate(b.get_m()), "t": st["t"], "steps": st["steps"], "rhs": st["rhs"],
                "max_dmdt": st["max_dmdt"]}
    eng = _engine(case)
    eng.set_h_ext(H_EXT)
    eng.set_m(state["m"])
    f = eng.eval_fields()
    rp, ci, K, G, D, V = eng.csr()
    nob, tri, nrm, sa = eng.boundary()
    eng.close()
    return {"H_total": f["H_total"], "phi": f["phi"], "row_ptr": rp, "col_idx": ci, "K": K, "G": G, "D": D,
            "volumes": V, "boundary": nob, "triangles": tri, "normals": nrm, "angles": sa}


# ---- what a pass cannot do without ----

def _counts(case):
    """(nodes, tetrahedra, nonzeros, boundary nodes) of a box."""
    a, b, c = case["nx"], case["ny"], case["nz"]
    n, t = (a + 1) * (b + 1) * (c + 1), 6 * a * b * c
    inner = max(0, a - 1) * max(0, b - 1) * max(0, c - 1)
    edges = (a * (b + 1) * (c + 1) + (a + 1) * b * (c + 1) + (a + 1) * (b + 1) * c) \
        + (a * b * (c + 1) + a * (b + 1) * c + (a + 1) * b * c) + a * b * c
    return n, t, n + 2 * edges, n - inner


def work(case):
    kind = case["kind"]
    if kind == "particles":
        r = 0.0
        for k in range(case["count"]):
            c = case["lo"] + int(round((case["hi"] - case["lo"]) * k / max(1, case["count"] - 1)))
            n, t, nnz, nb = _counts({"nx": c, "ny": c, "nz": c})
            r += 4.0 * nb * nb + 92.0 * nnz
        return {"bytes": 3.0 * case["launches"] * r, "flops": 0.5 * 3.0 * case["launches"] * r}
    n, t, nnz, nb = _counts(case)
    entry = {"fp64": 8.0, "fp32": 4.0, "fp32x2": 6.0, "bf16x3": 6.0}[case["form"]]
    # one right-hand side: the matrix, the gradient and divergence operators, the stiffness
    # twice (two Poisson solves, one pass over the operator each), m, H and dm/dt
    rhs_bytes = entry * nb * nb + nnz * (48.0 + 3 * 12.0) + 24.0 * 4 * n
    rhs_flops = 2.0 * nb * nb + nnz * 24.0 + 100.0 * n
    if kind == "fields":
        return {"bytes": case["count"] * rhs_bytes, "flops": case["count"] * rhs_flops}
    if kind == "advance":   # at least two right-hand sides for a start and one a record
        count = case["members"]
        chunk = -(-count // 8)
        evals = 2 + case["records"]
        return {"bytes": evals * (chunk * entry * nb * nb + count * (rhs_bytes - entry * nb * nb)),
                "flops": evals * count * rhs_flops}
    if kind == "product":
        r = case["rhs"]
        return {"bytes": entry * nb * nb + 16.0 * nb * r, "flops": (12.0 if case["form"] == "bf16x3" else 2.0) * nb * nb * r}
    if kind == "gradient":   # four stages forward, four recomputed, four transposed
        return {"bytes": 12.0 * case["steps"] * rhs_bytes, "flops": 12.0 * case["steps"] * rhs_flops}
    # setup: every (boundary node, outer triangle) pair takes about 250 operations
    faces = 4.0 * (case["nx"] * case["ny"] + case["ny"] * case["nz"] + case["nx"] * case["nz"])
    return {"bytes": 8.0 * nb * nb + 200.0 * nnz + rhs_bytes, "flops": 250.0 * nb * faces + rhs_flops}


# ---- the same in plain torch, 64 bits ----

class _Exact:
    """P1 operators, boundary matrix and field of a box, from the definitions."""

    def __init__(self, case):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        p, t = _box(case)
        self.p, self.t = torch.tensor(p, device=self.dev), torch.tensor(t, dtype=torch.int64, device=self.dev)
        self.N, self.T = len(p), len(t)
        x = self.p[self.t]
        e = x[:, 1:] - x[:, :1]
        det = torch.linalg.det(e)
        g = torch.linalg.inv(e).transpose(1, 2)
        self.dL = torch.cat([-g.sum(1, keepdim=True), g], 1)       # (T, 4, 3) gradients of the hat functions
        self.adet = det.abs()
        self.V = self.add(self.t, (self.adet / 24.0)[:, None].expand(-1, 4))
        row = self.t[:, :, None].expand(-1, 4, 4).reshape(-1)
        col = self.t[:, None, :].expand(-1, 4, 4).reshape(-1)
        k = torch.einsum("tad,tbd->tab", self.dL, self.dL) * (self.adet / 6.0)[:, None, None]
        self.K = torch.sparse_coo_tensor(torch.stack([row, col]), k.reshape(-1), (self.N, self.N)).coalesce()
        i = self.K.indices()
        self.diag = torch.zeros(self.N, dtype=torch.float64, device=self.dev)
        on = i[0] == i[1]
        self.diag[i[0][on]] = self.K.values()[on]
        self.Kc = self.K.to_sparse_csr()
        # outer faces: those of one tetrahedron only
        f = torch.cat([self.t[:, [a for a in range(4) if a != o]] for o in range(4)])
        s = f.sort(1).values
        key = (s[:, 0] * self.N + s[:, 1]) * self.N + s[:, 2]
        _, inv, cnt = torch.unique(key, return_inverse=True, return_counts=True)
        outer = cnt[inv] == 1
        self.face = f[outer]
        self.far = self.dL.transpose(0, 1).reshape(-1, 3)[outer]   # gradient of the opposite vertex: points inwards
        self.bnd = torch.unique(self.face)
        self.inner = torch.ones(self.N, dtype=torch.bool, device=self.dev)
        self.inner[self.bnd] = False

    def add(self, idx, val):
        out = torch.zeros((self.N,) + val.shape[2:], dtype=torch.float64, device=self.dev)
        return out.index_add(0, idx.reshape(-1), val.reshape((-1,) + val.shape[2:]))

    @staticmethod
    def omega(a, b, c):
        """Solid angle of a triangle seen from the origin."""
        la, lb, lc = a.norm(dim=-1), b.norm(dim=-1), c.norm(dim=-1)
        den = la * lb * lc + (a * b).sum(-1) * lc + (b * c).sum(-1) * la + (c * a).sum(-1) * lb
        return 2.0 * torch.atan2((a * torch.linalg.cross(b, c)).sum(-1).abs(), den)

    def bem(self):
        """Double-layer matrix (column c, observer k), transposed."""
        if hasattr(self, "Bt"):
            return self.Bt
        nb = len(self.bnd)
        of = torch.full((self.N,), -1, dtype=torch.int64, device=self.dev)
        of[self.bnd] = torch.arange(nb, device=self.dev)
        obs = self.p[self.bnd]
        Bt = torch.zeros(nb, nb, dtype=torch.float64, device=self.dev)
        eps = 1e-13 * float(self.p.abs().max())
        n = max(1, int(1.2e7 // nb))
        for c0 in range(0, len(self.face), n):
            face, far = self.face[c0:c0 + n], self.far[c0:c0 + n]
            q = self.p[face]                                       # (n, 3, 3)
            side = torch.stack([q[:, 2] - q[:, 1], q[:, 0] - q[:, 2], q[:, 1] - q[:, 0]], 1)
            sl = side.norm(dim=-1)
            xi = side / sl[..., None]
            z = torch.linalg.cross(side[:, 0], side[:, 1])
            area = 0.5 * z.norm(dim=-1)
            zh = z / z.norm(dim=-1, keepdim=True)
            eta = torch.linalg.cross(zh[:, None].expand(-1, 3, -1), xi)
            sign = torch.where((zh * far).sum(-1) > 0.0, -1.0, 1.0)   # the outward normal is against `far`
            gam = torch.einsum("nid,njd->nij", xi, xi)
            r = [q[:, v, None, :] - obs[None] for v in range(3)]   # (n, nb, 3)
            l = [v.norm(dim=-1) for v in r]
            pl = []
            for i in range(3):
                a, b, s = l[(i + 1) % 3], l[(i + 2) % 3], sl[:, i, None]
                pl.append(torch.log((a + b + s) / (a + b - s)))
            zeta = (zh[:, None] * r[0]).sum(-1)
            om = self.omega(*r)
            om = torch.where(zeta < 0.0, -om, om)
            good = (zeta.abs() > eps) & (l[0] > 0) & (l[1] > 0) & (l[2] > 0)
            fac = (sign * (sl.new_tensor(1.0) / (8.0 * math.pi * area)))[:, None]
            for i in range(3):
                e = torch.einsum("nd,nkd->nk", eta[:, i], r[(i + 1) % 3])
                gl = gam[:, i, 0, None] * pl[0] + gam[:, i, 1, None] * pl[1] + gam[:, i, 2, None] * pl[2]
                val = fac * sl[:, i, None] * (om * e - zeta * gl)
                Bt.index_add_(0, of[face[:, i]], torch.where(good, val, torch.zeros_like(val)))
        ang = torch.zeros(self.N, dtype=torch.float64, device=self.dev)
        for a in range(4):
            o = [b for b in range(4) if b != a]
            d = [self.p[self.t[:, b]] - self.p[self.t[:, a]] for b in o]
            ang.index_add_(0, self.t[:, a], self.omega(*d))
        self.angle = ang[self.bnd]
        Bt.diagonal().add_(self.angle / (4.0 * math.pi) - 1.0)
        self.Bt = Bt
        return Bt

    def solve(self, b, neumann):
        """K x = b for every column of b: mean-free, or on the inner nodes alone."""
        keep = None if neumann else self.inner.double()[:, None]
        b = b - b.mean(0) if neumann else b * keep
        x, r = torch.zeros_like(b), b.clone()
        z = r / self.diag[:, None]
        p, rz = z.clone(), (r * z).sum(0)
        tol = (b * b).sum(0).clamp_min(1e-300) * 1e-30
        best = torch.full_like(rz, math.inf)
        for it in range(6000):
            q = self.Kc @ p
            if keep is not None:
                q = q * keep
            al = rz / (p * q).sum(0).clamp_min(1e-300)
            x += al * p
            r -= al * q
            if it % 20 == 19:
                rr = (r * r).sum(0)
                if bool((rr <= tol).all()) or bool((rr > 1e6 * best).any()):
                    break
                best = torch.minimum(best, rr)
            z = r / self.diag[:, None]
            new = (r * z).sum(0)
            p = z + (new / rz.clamp_min(1e-300)) * p
            rz = new
        return x - x.mean(0) if neumann else x

    def charges(self, m, wD=None):
        """Ms int M . grad of every hat function, for states m (N, 3, R)."""
        s = m[self.t].sum(1) * (MS * self.adet / 24.0 * (1.0 if wD is None else wD))[:, None, None]
        return self.add(self.t, torch.einsum("tad,tdr->tar", self.dL, s))

    def potential(self, rho):
        phi1 = self.solve(rho, True)
        pb = self.bem().T @ phi1[self.bnd]
        full = torch.zeros_like(phi1)
        full[self.bnd] = pb
        return phi1 + full + self.solve(-(self.Kc @ full), False)

    def minus_grad(self, phi):
        g = torch.einsum("tbd,tbr->tdr", self.dL, phi[self.t]) * (self.adet / 24.0)[:, None, None]
        return -self.add(self.t, g[:, None].expand(-1, 4, -1, -1)) / self.V[:, None, None]

    def exchange(self, m, wK=None):
        g = torch.einsum("tbd,tbcr->tdcr", self.dL, m[self.t])
        w = self.adet / 6.0 * (1.0 if wK is None else wK)
        k = torch.einsum("tad,tdcr->tacr", self.dL, g) * w[:, None, None, None]
        return -C_EXCH * self.add(self.t, k) / self.V[:, None, None]


def _llg(m, H):
    """dm/dt of states and fields (N, 3, R)."""
    mxH = torch.linalg.cross(m, H, dim=1)
    return -0.221012 * mxH - 0.00442023 * torch.linalg.cross(m, mxH, dim=1) \
        + 0.1 * (1.0 - (m * m).sum(1, keepdim=True)) * m


def _exact_fields(ex, case, states):
    m = torch.tensor(np.stack(states, -1), device=ex.dev)
    phi = ex.potential(ex.charges(m))
    hd, hx = ex.minus_grad(phi), ex.exchange(m)
    ha = torch.zeros_like(m)
    axis = torch.tensor(AXIS, dtype=torch.float64, device=ex.dev)
    he = torch.tensor(H_EXT, dtype=torch.float64, device=ex.dev)[None, :, None]
    anis = case.get("anis", 0.0)
    am = torch.einsum("d,ndr->nr", axis, m)[:, None]
    if anis:
        ha = 2.0 * anis / (1.2566370614 * MS) * am * (axis[None, :, None] - am * m)
    H = he + hx + ha + hd
    dens = torch.stack([-0.540354 * (m * hx).sum(1), -0.540354 * (m * hd).sum(1), -1.08071 * (m * he).sum(1),
                        -anis * am[:, 0] ** 2])
    en = (dens * ex.V[None, :, None]).sum(1)
    return H, _llg(m, H), torch.cat([en, en.sum(0, keepdim=True)]), phi


def _exact_gradient(ex, case, seed):
    d = {k: torch.tensor(v, dtype=torch.float64, device=ex.dev).requires_grad_(True)
         for k, v in _gradient_inputs(case, ex.N, ex.T, seed).items()}
    # phi is linear in the charges: the dense map once, from unit charges
    L = ex.potential(torch.eye(ex.N, dtype=torch.float64, device=ex.dev))
    wK, wD = MS / d["Ms"], d["Ms"] / MS
    kap = 2.0 * d["K1"] / (1.2566370614 * d["Ms"])
    c = ex.add(ex.t, (ex.adet / 24.0 * kap)[:, None].expand(-1, 4)) / ex.V
    axis = torch.tensor(AXIS, dtype=torch.float64, device=ex.dev)
    he = torch.tensor(H_EXT, dtype=torch.float64, device=ex.dev)
    spp = max(1, case["steps"] // case["pulses"])

    def f(m, n):
        h = he + (d["pulses"][n // spp] if n // spp < case["pulses"] else 0.0)
        am = torch.einsum("d,ndr->nr", axis, m)[:, None]
        H = h[None, :, None] + ex.exchange(m, wK) + c[:, None, None] * am * (axis[None, :, None] - am * m) \
            + ex.minus_grad(L @ ex.charges(m, wD))
        return _llg(m, H)

    m, hist = d["m0"].reshape(-1, 3, 1), []
    for n in range(case["steps"]):
        k1 = f(m, n)
        k2 = f(m + 0.05 * k1, n)
        k3 = f(m + 0.05 * k2, n)
        k4 = f(m + 0.1 * k3, n)
        m = m + (0.1 / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        hist.append((m[:, :, 0] * ex.V[:, None]).sum(0) / ex.V.sum())
    hist = torch.stack(hist)
    target = torch.tensor((0.0, 1.0, 0.0), dtype=torch.float64, device=ex.dev)
    loss = ((hist[-1] - target) ** 2).sum() + 1e-3 * (hist[:, 0] ** 2).mean()
    g = torch.autograd.grad(loss, [d[k] for k in ("m0", "Ms", "K1", "pulses")])
    return {"m": m.detach().reshape(-1), "history": hist.detach(), "loss": loss.detach(), "gradients": list(g)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("advance", "particles"):   # whole integrations: no closed result
        return None
    if kind == "gradient" and _counts(case)[0] > 2500:
        return None
    ex = _Exact(case)
    if kind == "product":
        x = torch.tensor(_potentials(case, len(ex.bnd), seed), device=ex.dev)
        return x @ ex.bem()
    if kind == "gradient":
        return _exact_gradient(ex, case, seed)
    if kind == "fields":
        H, f, en, _ = _exact_fields(ex, case, _states(case, ex.N, seed))
        n = range(case["count"])
        return {"H_total": [H[:, :, k].contiguous() for k in n], "dmdt": [f[:, :, k].contiguous() for k in n],
                "energies": [en[:, k].contiguous() for k in n]}
    H, _, _, phi = _exact_fields(ex, case, _states({"count": 1}, ex.N, seed))
    none = ("row_ptr", "col_idx", "K", "G", "D", "boundary", "triangles", "normals")
    return dict({k: None for k in none}, H_total=H[:, :, 0].contiguous(), phi=phi[:, 0].contiguous(), volumes=ex.V,
                angles=ex.angle)
