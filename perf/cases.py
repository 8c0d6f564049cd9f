"""Performance cases of the assembly path: the calls a program built on pigfem_b200 makes.

A case names a mesh (element type, grid, inclusions, interface law, loading), the call made on it
and its options.  The kinds of call:

* ``tangent``   one device assembly (K and R, or R alone, FP64 or FP32-mixed) of a resident RVE;
* ``newton``    a Newton iteration's share: K and R, then the residual norm the solver tests;
* ``strains``   a linear periodic RVE's K and R plus the residuals of the other unit strains;
* ``host``      the drop-in call on host buffers (U up, residuals and changed K values back);
* ``batch``     several RVEs of uneven size in one batched assembly;
* ``solve``     Jacobi-PCG on an assembled K_ff with several right-hand sides;
* ``request``   a whole homogenization request: K, unit-strain residuals, solve, averages.

The meshes are seeded fiber composites with the constants of pigfem_b200.rve, their sizes those of
bench.py's workloads and the serving stream's request ranges (2D 32^2 to 512^2 with 5 to 300
fibers, 3D 16^3 to 64^3 with 5 to 60 spheres).  A case's mesh is fixed by its ``layout``; the seed
draws the displacement state, the materials or the right-hand sides.
"""
import math

import numpy as np
import torch

from pigfem_b200 import capi, rve

TRI3, QUAD4, TET4 = "tri3", "quad4", "tet4"
_TYPE = {TRI3: capi.TRI3, QUAD4: capi.QUAD4, TET4: capi.TET4}
_LAW = {"none": (capi.COH_NONE, (0.0,) * 4), "bilinear": (capi.COH_BL, rve.BL_PARAMS),
        "ortiz": (capi.COH_OP, (50.0, 2e-4, 1.0, 0.0))}
_RTOL = 1e-12     # close to the Newton corrections' 1e-13, so that two solvers' results can be compared


def _case(kind, elem, n, incl, vf, law="none", periodic=False, **kw):
    c = {"kind": kind, "elem": elem, "nx": n[0], "ny": n[1], "nz": n[2] if len(n) > 2 else 0, "inclusions": incl,
         "volume_fraction": vf, "law": law, "periodic": periodic, "layout": 1}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest mesh of the serving stream inside a Newton loop: latency and launches
        dict(_case("newton", TRI3, (32, 32), 6, 0.12, "bilinear"), name="newton_2d_32"),
        # the linear 2D RVE (64 x 64, ten fibers, prescribed strain): K and R once
        dict(_case("tangent", TRI3, (64, 64), 10, 0.06), name="linear_2d_64"),
        # the headline workload: 512 x 512, 200 fibers, bilinear interfaces, FP64
        dict(_case("tangent", TRI3, (512, 512), 200, 0.085, "bilinear"), name="cohesive_2d_512"),
        # the FP32-mixed option, on a ragged grid with hx != hy
        dict(_case("tangent", TRI3, (301, 187), 60, 0.15, "bilinear", fp32=True), name="cohesive_2d_301x187_fp32"),
        # R alone (a line search, a load case of a fixed K), interfaces with damage memory
        dict(_case("tangent", TRI3, (397, 400), 150, 0.2, "ortiz", residual_only=True), name="residual_2d_397x400"),
        # quad4 background elements, cut and uncut
        dict(_case("tangent", QUAD4, (200, 150), 40, 0.15, "bilinear"), name="quad4_2d_200x150"),
        # a 3D cohesive load step of a small ragged grid
        dict(_case("tangent", TET4, (22, 18, 25), 6, 0.04, "bilinear"), name="cohesive_3d_22x18x25"),
        # the 3D benchmark step: 64^3 hexes in six tets, 50 spheres, K once and six unit strains
        dict(_case("strains", TET4, (64, 64, 64), 50, 0.045, periodic=True), name="strains_3d_64"),
        # uneven 2D RVEs assembled together (the batched workload's size range)
        dict(_case("batch", TRI3, (32, 256), 40, 0.3, "bilinear", count=10), name="batch_2d_10"),
        # the six load cases of a 3D homogenization solved together
        dict(_case("solve", TET4, (40, 40, 40), 20, 0.03, periodic=True, rhs=6), name="solve_3d_40"),
        # a whole 2D homogenization request
        dict(_case("request", TRI3, (128, 128), 60, 0.2, periodic=True), name="request_2d_128"),
        # the drop-in call on host buffers, as a host solver's Newton loop makes it
        dict(_case("host", TRI3, (256, 256), 80, 0.15, "bilinear"), name="host_2d_256"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["newton", "tangent", "tangent", "tangent", "strains", "host", "batch", "solve", "request"])
    three_d = kind in ("tangent", "strains", "solve", "request") and rng.random() < 0.4
    layout = rng.randrange(1, 1000)
    if kind == "batch":
        return _case("batch", TRI3, (32, size(64, 256)), rng.randint(10, 60), rng.uniform(0.2, 0.4), "bilinear",
                     count=rng.randint(3, 10), layout=layout, fp32=rng.random() < 0.5)
    if three_d:
        hi = {"tangent": 48, "strains": 56, "solve": 36, "request": 28}[kind]
        n = [size(16, hi)] * 3 if rng.random() < 0.3 else [size(16, hi) for _ in range(3)]
        c = _case(kind, TET4, n, rng.randint(5, 12 if min(n) < 24 else 30), rng.uniform(0.02, 0.04), layout=layout,
                  periodic=kind != "tangent")
    else:
        hi = {"newton": 512, "tangent": 512, "strains": 512, "host": 300, "solve": 256, "request": 160}[kind]
        n = [size(32, hi)] * 2
        if rng.random() < 0.6:
            n[1] = max(32, int(n[0] * rng.uniform(0.5, 1.0)))
        c = _case(kind, TRI3, n, rng.randint(5, max(6, min(300, n[1] * n[1] // 150))), rng.uniform(0.06, 0.25), layout=layout,
                  periodic=kind in ("strains", "solve", "request"))
        if kind == "tangent" and rng.random() < 0.25:
            c["elem"] = QUAD4
            c["nx"], c["ny"] = min(c["nx"], 256), min(c["ny"], 256)
    if kind in ("newton", "tangent", "host") and rng.random() < 0.8:
        c["law"] = rng.choice(["bilinear", "ortiz"])
    if kind == "tangent":
        c["fp32"] = rng.random() < 0.25
        c["residual_only"] = rng.random() < 0.25
    if kind == "solve":
        c["rhs"] = 6 if c["elem"] == TET4 else rng.choice([1, 3])
    return c


# ------------------------------------------------------------------ meshes and states
def _describe(c, attempt, seed=None, sub=0):
    """The case's RVE: seeded non-overlapping circles / spheres in the unit box with radii
    0.8 to 1.2 of the mean radius the volume fraction asks for.  With a seed, seeded materials."""
    dim = 3 if c["elem"] == TET4 else 2
    n = [c["nx"], c["ny"], c["nz"]][:dim]
    nf, vf = c["inclusions"], c["volume_fraction"]
    rng = rve.philox(17 + sub, c["layout"], attempt)
    if c["kind"] == "batch":
        side = int(round(math.exp(rng.uniform(math.log(c["nx"]), math.log(c["ny"])))))
        n = [side, side]
        nf = int(rng.integers(5, nf + 1))
    h = 1.0 / min(n)
    if dim == 2:
        r = math.sqrt(vf / (nf * math.pi))
        gap, accept = 0.002, None
    else:
        r = (vf / (nf * 4.0 / 3.0 * math.pi)) ** (1.0 / 3.0)
        # no tet may see two spheres; a sphere whose top lies above cy + r may be cut off by the
        # reference's bounding box, so its centre keeps to z <= y
        gap, accept = max(0.01, 1.8 * h), (lambda x, _r: x[2] <= x[1])
    incl = rve.place_fibers(rng, nf, 0.8 * r, 1.2 * r, gap, dim, max_attempts=4000, accept=accept)
    law, par = _LAW[c["law"]]
    s = np.ones(2) if seed is None else np.random.default_rng(seed).uniform(0.8, 1.2, 2)
    eps = ((1.0, 0.0, 0.0) if dim == 2 else (1.0, 0.0, 0.0, 0.0, 0.0, 0.0)) if c["periodic"] else (0.0,) * 6
    return capi.ProblemDesc(elem_type=_TYPE[c["elem"]], n=n, lo=(0.0,) * dim, hi=(1.0,) * dim, inclusions=incl,
                            E_matrix=rve.E_MATRIX * s[0], nu_matrix=rve.NU_MATRIX, E_fiber=rve.E_FIBER * s[1],
                            nu_fiber=rve.NU_FIBER, coh_law=law, coh=par, plane_strain=True, subscale=c["periodic"],
                            eps_macro=eps, app_strain=0.02)


def _problem(c, seed=None, sub=0, device=True):
    """The first admissible layout (a grid node on an interface or an element seeing too many
    inclusions is refused by the set-up, as by the reference)."""
    for attempt in range(40):
        try:
            return capi.Problem(_describe(c, attempt, seed, sub), device=device)
        except capi.PigfemError as e:
            if e.code not in (3, 4):
                raise
    raise RuntimeError("no admissible layout")


def _displacements(p, c, seed):
    """Interfaces opened through the law's branches; without interfaces a random field of 1e-3."""
    if c["law"] == "none":
        return np.random.default_rng(seed).uniform(-1e-3, 1e-3, p.n_nodes * p.dim)
    return rve.interface_state(p, seed=seed, open_lo=1e-7, open_hi=6e-3 if c["law"] == "bilinear" else 1e-3)


def _fluctuation(p, seed):
    """A random field of the DOFs (a node's periodic images share its values), node-major."""
    _, dofs, _ = p.nodes()
    return np.random.default_rng(seed).uniform(-1e-3, 1e-3, p.n_free + p.n_const)[dofs.reshape(-1)]


def _flags(c):
    f = capi.FUNC if c.get("residual_only") else capi.FUNC | capi.JAC
    return f | (capi.FP32 if c.get("fp32") else 0)


def _views(p):
    """The context's device outputs as tensors that keep the context alive."""
    K, pf, pp = p.device_outputs()
    v = {"K_" + b: capi.device_view(K[i], p.nnz[i]) for i, b in enumerate(("ff", "fp", "pf", "pp")) if p.nnz[i]}
    v["P_f"] = capi.device_view(pf, p.n_free)
    if p.n_const:
        v["P_p"] = capi.device_view(pp, p.n_const)
    for t in v.values():
        t.context = p
    return v


def _units(p):
    nv = 3 if p.dim == 2 else 6
    return [list(row) for row in np.eye(nv)]


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "batch":
        ps = [_problem(c, sub=i) for i in range(c["count"])]
        u = [torch.from_numpy(_displacements(p, c, seed + 31 * i)).cuda() for i, p in enumerate(ps)]
        return {"case": c, "p": ps, "u": u, "batch": capi.Batch(ps), "out": [_views(p) for p in ps]}
    p = _problem(c, seed if k in ("strains", "request") else None)
    st = {"case": c, "p": p}
    if k in ("tangent", "newton"):
        st["u"] = torch.from_numpy(_displacements(p, c, seed)).cuda()
        v = _views(p)
        st["out"] = {n: t for n, t in v.items() if n.startswith("P")} if c.get("residual_only") else v
    elif k == "host":
        def pinned(n):
            return torch.zeros(max(1, n), dtype=torch.float64, pin_memory=True).numpy()
        st["u"] = pinned(p.n_nodes * p.dim)
        st["u"][:] = _displacements(p, c, seed)
        st["out"] = {"K_" + b: pinned(p.nnz[i]) for i, b in enumerate(("ff", "fp", "pf", "pp"))}
        st["out"].update(P_f=pinned(p.n_free), P_p=pinned(p.n_const))
    else:
        nv = len(_units(p))
        n = p.n_free
        zero = np.zeros(p.n_nodes * p.dim)
        st["zero"] = torch.from_numpy(zero).cuda()
        if k == "strains":
            # the field of the first load case's last iterate: a small random fluctuation
            st["u"] = torch.from_numpy(_fluctuation(p, seed + 1)).cuda()
            st["out"] = _views(p)
        if k in ("strains", "request"):
            st["rf"] = torch.empty(nv * n, dtype=torch.float64, device="cuda")
            st["rp"] = torch.empty(max(1, nv * p.n_const), dtype=torch.float64, device="cuda")
        if k == "request":
            st["x"] = torch.empty(nv * n, dtype=torch.float64, device="cuda")
            _, dofs, _ = p.nodes()
            st["dofs"] = torch.from_numpy(dofs.reshape(-1).astype(np.int64)).cuda()
        if k == "solve":
            p.assemble_device(st["zero"].data_ptr(), 1.0, capi.JAC)
            b = np.random.default_rng(seed).uniform(-1.0, 1.0, c["rhs"] * n)
            st["b"] = torch.from_numpy(b).cuda()
            st["x"] = torch.empty_like(st["b"])
    return st


def run(state):
    c, p = state["case"], state["p"]
    k = c["kind"]
    if k == "tangent":
        p.assemble_device(state["u"].data_ptr(), 1.0, _flags(c))
        return state["out"]
    if k == "newton":
        p.assemble_device(state["u"].data_ptr(), 1.0, _flags(c))
        return dict(state["out"], norm=p.residual_norm())
    if k == "batch":
        state["batch"].assemble([u.data_ptr() for u in state["u"]], _flags(c))
        state["batch"].wait()
        return state["out"]
    if k == "host":
        return p.assemble(state["u"], 1.0, _flags(c) | capi.KEEP_STATIC, out=state["out"])
    units = _units(p)
    if k == "strains":
        p.assemble_device(state["u"].data_ptr(), 1.0, capi.FUNC | capi.JAC)
        p.residual_strains(state["u"].data_ptr(), units[1:], state["rf"].data_ptr(), state["rp"].data_ptr())
        m = len(units) - 1
        return dict(state["out"], cases_f=state["rf"][:m * p.n_free], cases_p=state["rp"][:m * p.n_const])
    if k == "solve":
        state["x"].zero_()
        p.pcg_solve(state["b"].data_ptr(), state["x"].data_ptr(), c["rhs"], _RTOL)
        return state["x"]
    # a homogenization request, as the serving loop runs it
    n, nv = p.n_free, len(units)
    p.assemble_device(state["zero"].data_ptr(), 1.0, capi.JAC)
    p.residual_strains(state["zero"].data_ptr(), units, state["rf"].data_ptr(), state["rp"].data_ptr())
    state["x"].zero_()
    p.pcg_solve(state["rf"].data_ptr(), state["x"].data_ptr(), nv, _RTOL)
    C = np.zeros((nv, nv))
    full = torch.zeros(n + p.n_const, dtype=torch.float64, device="cuda")
    for j, e in enumerate(units):
        p.set_macro_strain(e)
        full[:n] = -state["x"][j * n:(j + 1) * n]
        u = full[state["dofs"]]
        C[:, j] = p.homogenize(u.data_ptr(), 1.0)[:nv]
    return {"x": state["x"], "C": C}


# ------------------------------------------------------------------ the work of a pass
def work(case):
    """Bytes: U, the elements' material tags and the cohesive points' tables read once, K and R
    written once (what the cut elements' points need is left out).  The host call adds the copies
    of U, of the residuals and of the K values that can change.  A solve reads the matrix (values
    and columns) and five vectors and writes three per right-hand side and iteration; its
    iteration count is taken as 25 times the longest grid side."""
    c, k = case, case["kind"]
    ps = [_problem(c, sub=i, device=False) for i in range(c.get("count", 1))] if k == "batch" else [_problem(c, device=False)]
    total = flops = 0.0
    for p in ps:
        s = p.sizes
        dim, npe = p.dim, 4 if c["elem"] != TRI3 else 3
        nv = 3 if dim == 2 else 6
        nnz, rows = sum(s["nnz"]), s["n_free"] + s["n_const"]
        state = 8 * dim * s["n_nodes"] + 4 * s["n_elem"] + 16 * s["n_isv"] + 8 * s["n_coh_qp"] * (dim * dim + 3)
        resid = 8 * rows
        nd = npe * dim
        if k in ("tangent", "newton", "batch"):
            jac = not c.get("residual_only")
            total += state + resid + (8 * nnz if jac else 0)
            flops += s["n_elem"] * ((nd * nd if jac else 0) + 4 * nd * nv)
        elif k == "strains":
            total += state + 8 * nnz + nv * resid
            flops += s["n_elem"] * (nd * nd + nv * 4 * nd * nv)
        elif k == "host":
            changed = sum(z - f for z, f in zip(s["nnz"], p.changing_values())) if s["n_isv"] else 0
            total += state + 2 * resid + 8 * (nnz + max(0, changed))
            flops += s["n_elem"] * (nd * nd + 4 * nd * nv)
        else:
            rhs = c.get("rhs", nv)
            iters = 25 * max(c["nx"], c["ny"], c["nz"])
            total += iters * (12.0 * s["nnz"][0] + 64.0 * rhs * s["n_free"])
            flops += iters * rhs * (2.0 * s["nnz"][0] + 12.0 * s["n_free"])
            if k == "request":
                total += state + 8 * nnz + nv * (resid + state)
                flops += s["n_elem"] * (nd * nd + 2 * nv * 4 * nd * nv)
        p.close()
    return {"bytes": float(total), "flops": float(flops)}


# ------------------------------------------------------------------ the same values in plain torch
class _Exact:
    """K, P and volume averages in 64-bit torch from the enriched mesh's own tables (coordinates,
    connectivity, sub-element points with their gradients and weights, cohesive points), which the
    set-up hands to any assembler; the integrals, laws and scatter are formed here."""

    def __init__(self, p, c):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.dim, self.nf, self.nc = p.dim, p.n_free, p.n_const
        self.nv = 3 if p.dim == 2 else 6
        d, dim = p.desc, p.dim
        X, dofs, _ = p.nodes()
        self.X, self.dof = self.t(X), self.t(dofs.astype(np.int64))
        self.conn = self.t(p.debug("conn").astype(np.int64)).reshape(p.sizes["n_elem"], -1)
        self.emat = self.t(p.debug("elem_mat").astype(np.int64))
        self.cut = self.t(p.debug("cut_of").astype(np.int64)) >= 0
        self.D = torch.stack([self.t(self.elastic(E, nu)) for E, nu in
                              ((d.E_matrix, d.nu_matrix), (d.E_fiber, d.nu_fiber))])
        g = {k: p.debug(k) for k in ("cut_node_off", "cut_nodes", "cut_qp_off", "qp_wgt", "qp_mat", "qp_grad_off", "qp_grad",
                                     "cut_coh_off", "coh_nh", "coh_local_off", "coh_local", "coh_qp_off", "cqp_N",
                                     "cqp_R", "cqp_wgt")}
        self.groups = list(self.uncut()) + list(self.cut_groups(g))
        self.coh = list(self.cohesive(g)) if c["law"] != "none" else []
        self.law, self.par = c["law"], _LAW[c["law"]][1]
        self.pat = [p.pattern(b) for b in range(4)]

    def t(self, a):
        return torch.as_tensor(np.ascontiguousarray(a), device=self.dev)

    def elastic(self, E, nu):
        f = E / ((1.0 + nu) * (1.0 - 2.0 * nu))
        D = np.zeros((self.nv, self.nv))
        D[:self.dim, :self.dim] = f * nu
        D[range(self.dim), range(self.dim)] = f * (1.0 - nu)
        D[range(self.dim, self.nv), range(self.dim, self.nv)] = f * (1.0 - 2.0 * nu) / 2.0
        return D

    def strain_matrix(self, g):
        """B of point gradients g (..., nodes, dim), engineering shear in the order yz, xz, xy."""
        B = torch.zeros(g.shape[:-2] + (self.nv, g.shape[-2], self.dim), dtype=torch.float64, device=self.dev)
        for i in range(self.dim):
            B[..., i, :, i] = g[..., i]
        for r, (i, j) in enumerate([(0, 1)] if self.dim == 2 else [(1, 2), (0, 2), (0, 1)]):
            B[..., self.dim + r, :, i] = g[..., j]
            B[..., self.dim + r, :, j] = g[..., i]
        return B.flatten(-2)

    def uncut(self):
        """(nodes, gradients, weights, materials) of the uncut elements, a set per Gauss point."""
        conn, mat = self.conn[~self.cut], self.emat[~self.cut]
        if conn.shape[1] == self.dim + 1:
            ref = torch.cat([-torch.ones(1, self.dim), torch.eye(self.dim)]).double().to(self.dev)
            pts, w = [ref], [0.5 if self.dim == 2 else 1.0]      # the reference's tet weights sum to one
        else:
            a = 1.0 / math.sqrt(3.0)
            pts, w = [], [1.0] * 4
            for r, s in ((-a, -a), (a, -a), (-a, a), (a, a)):
                pts.append(0.25 * torch.tensor([[-(1 - s), -(1 - r)], [1 - s, -(1 + r)], [1 + s, 1 + r], [-(1 + s), 1 - r]],
                                               dtype=torch.float64, device=self.dev))
        step = 100000
        for a in range(0, len(conn), step):
            nodes = conn[a:a + step]
            x = self.X[nodes]
            for dN, wq in zip(pts, w):
                J = torch.einsum("na,eni->eai", dN, x)
                g = torch.einsum("na,eia->eni", dN, torch.linalg.inv(J))
                yield nodes, g, wq * torch.linalg.det(J), mat[a:a + step]

    def cut_groups(self, g):
        off, qoff, goff = g["cut_node_off"], g["cut_qp_off"], g["qp_grad_off"]
        nn, nq = np.diff(off), np.diff(qoff)
        el = np.repeat(np.arange(len(nq)), nq)                    # element of each point
        for m in np.unique(nn):
            q = np.nonzero(nn[el] == m)[0]
            for a in range(0, len(q), 200000):
                s = q[a:a + 200000]
                nodes = g["cut_nodes"][off[el[s]][:, None] + np.arange(m)]
                grad = g["qp_grad"][goff[s][:, None] + np.arange(m * self.dim)].reshape(-1, m, self.dim)
                yield (self.t(nodes.astype(np.int64)), self.t(grad), self.t(g["qp_wgt"][s]),
                       self.t(g["qp_mat"][s].astype(np.int64)))

    def cohesive(self, g):
        nq, nh = np.diff(g["coh_qp_off"]), g["coh_nh"]
        ce_cut = np.repeat(np.arange(len(g["cut_coh_off"]) - 1), np.diff(g["cut_coh_off"]))
        el = np.repeat(np.arange(len(nq)), nq)
        noff = np.concatenate([[0], np.cumsum(nh[el])])[:-1]
        R = g["cqp_R"].reshape(-1, self.dim, self.dim)
        for h in np.unique(nh):
            q = np.nonzero(nh[el] == h)[0]
            e = el[q]
            loc = g["coh_local"][g["coh_local_off"][e][:, None] + np.arange(2 * h)]
            nodes = g["cut_nodes"][g["cut_node_off"][ce_cut[e]][:, None] + loc]
            N = g["cqp_N"][noff[q][:, None] + np.arange(h)]
            yield (self.t(nodes.astype(np.int64)), self.t(np.concatenate([-N, N], axis=1)), self.t(R[q]),
                   self.t(g["cqp_wgt"][q]))

    def traction(self, dl):
        """Traction and tangent of tensile openings on the loading branch (no committed damage):
        effective opening sqrt(delta . delta), the bilinear or the exponential curve."""
        d = torch.linalg.norm(dl, dim=1)
        s, p1, p2 = self.par[0], self.par[1], self.par[2]
        if self.law == "bilinear":
            rise, fall = d < p1, (d >= p1) & (d < p2)
            t = torch.where(rise, d * (s / p1), torch.where(fall, s * (1 - (d - p1) / (p2 - p1)), 0 * d))
            dt = torch.where(rise, 0 * d + s / p1, torch.where(fall, 0 * d - s / (p2 - p1), 0 * d))
        else:
            t = s * (d / p1) * torch.exp(1.0 - d / p1)
            dt = (s / p1) * (1.0 - d / p1) * torch.exp(1.0 - d / p1)
        n = dl / d[:, None]
        nn = n[:, :, None] * n[:, None, :]
        eye = torch.eye(self.dim, dtype=torch.float64, device=self.dev)
        return t[:, None] * n, dt[:, None, None] * nn + (t / d)[:, None, None] * (eye - nn)

    def parts(self, u=None, strains=(), stiffness=True):
        """Per group: element DOFs, element matrices (or None), element forces per strain case."""
        for nodes, g, w, m in self.groups:
            B, D = self.strain_matrix(g), self.D[m]
            DB = torch.einsum("evw,ewi->evi", D, B)
            K = torch.einsum("e,evi,evj->eij", w, B, DB) if stiffness else None
            f = []
            if len(strains):
                e0 = torch.einsum("evi,ei->ev", B, u[nodes].flatten(1))
                for s in strains:
                    sig = torch.einsum("evw,ew->ev", D, e0 + self.t(np.asarray(s)))
                    f.append(torch.einsum("e,evi,ev->ei", w, B, sig))
            yield self.dof[nodes].flatten(1), K, f
        for nodes, N, R, w in self.coh:
            jump = torch.einsum("en,end->ed", N, u[nodes])
            T, Dc = self.traction(torch.einsum("eij,ej->ei", R, jump))
            K = None
            if stiffness:
                W = torch.einsum("e,eji,ejk,ekl->eil", w, R, Dc, R)
                K = torch.einsum("ea,eb,eil->eaibl", N, N, W).reshape(len(w), N.shape[1] * self.dim, -1)
            f = torch.einsum("e,ea,eji,ej->eai", w, N, R, T).flatten(1)
            yield self.dof[nodes].flatten(1), K, [f] * len(strains)

    def assemble(self, u=None, strains=(), stiffness=True):
        u = None if u is None else self.t(u).reshape(-1, self.dim)
        nt = self.nf + self.nc
        F = torch.zeros(len(strains), nt, dtype=torch.float64, device=self.dev)
        keys, vals = [], []
        if stiffness:
            for rp, ci, shape in self.pat:
                rows = torch.repeat_interleave(torch.arange(shape[0], device=self.dev), self.t(np.diff(rp).astype(np.int64)))
                keys.append(rows * shape[1] + self.t(ci.astype(np.int64)))
                vals.append(torch.zeros(len(ci), dtype=torch.float64, device=self.dev))
        for dof, K, f in self.parts(u, strains, stiffness):
            for s, fs in enumerate(f):
                F[s].index_add_(0, dof.flatten(), fs.flatten())
            if not stiffness:
                continue
            r, cc = (a.flatten() for a in torch.broadcast_tensors(dof[:, :, None], dof[:, None, :]))
            v = K.flatten()
            for b in range(4):
                if not len(vals[b]):
                    continue
                sel = ((r >= self.nf) == (b >= 2)) & ((cc >= self.nf) == (b % 2 == 1))
                rb, cb = r[sel] - (self.nf if b >= 2 else 0), cc[sel] - (self.nf if b % 2 else 0)
                vals[b].index_add_(0, torch.searchsorted(keys[b], rb * self.pat[b][2][1] + cb), v[sel])
        return vals, F

    def average(self, u, strain):
        u = u.reshape(-1, self.dim)
        tot, vol = torch.zeros(self.nv, dtype=torch.float64, device=self.dev), 0.0
        for nodes, g, w, m in self.groups:
            e = torch.einsum("evi,ei->ev", self.strain_matrix(g), u[nodes].flatten(1)) + self.t(np.asarray(strain))
            tot += torch.einsum("e,evw,ew->v", w, self.D[m], e)
            vol += float(w.sum())
        return (tot / vol).cpu().numpy()

    def solve(self, kff, b):
        """K_ff x = b by Jacobi-preconditioned conjugate gradients to 1e-13 (b: rhs x n)."""
        rp, ci, shape = self.pat[0]
        A = torch.sparse_csr_tensor(self.t(rp.astype(np.int64)), self.t(ci.astype(np.int64)), kff, size=shape)
        rows = torch.repeat_interleave(torch.arange(shape[0], device=self.dev), self.t(np.diff(rp).astype(np.int64)))
        dinv = 1.0 / kff[rows == self.t(ci.astype(np.int64))]
        B = b.t().contiguous()
        x, r = torch.zeros_like(B), B.clone()
        z = dinv[:, None] * r
        q = z.clone()
        rz, nb = (r * z).sum(0), torch.linalg.norm(B, dim=0)
        for k in range(20000):
            Aq = A @ q
            al = rz / (q * Aq).sum(0)
            x += al * q
            r -= al * Aq
            if k % 25 == 0 and float((torch.linalg.norm(r, dim=0) / nb).max()) < 1e-13:
                break
            z = dinv[:, None] * r
            new = (r * z).sum(0)
            q = z + (new / rz) * q
            rz = new
        return x.t().contiguous()


def _named(p, vals, F):
    out = {"K_" + b: v for b, v in zip(("ff", "fp", "pf", "pp"), vals) if len(v)}
    if len(F):
        out["P_f"] = F[0][:p.n_free]
        if p.n_const:
            out["P_p"] = F[0][p.n_free:]
    return out


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "batch":
        out = []
        for i in range(c["count"]):
            p = _problem(c, sub=i, device=False)
            vals, F = _Exact(p, c).assemble(_displacements(p, c, seed + 31 * i), [[0.0] * 3])
            out.append(_named(p, vals, F))
            p.close()
        return out
    p = _problem(c, seed if k in ("strains", "request") else None, device=False)
    E = _Exact(p, c)
    units = _units(p)
    if k in ("tangent", "newton", "host"):
        vals, F = E.assemble(_displacements(p, c, seed), [[0.0] * E.nv], not c.get("residual_only"))
        out = _named(p, vals, F)
        if k == "host":
            out = {n: v.cpu().numpy() for n, v in out.items()}
            for i, b in enumerate(("ff", "fp", "pf", "pp")):
                out.setdefault("K_" + b, np.zeros(0))
            out.setdefault("P_p", np.zeros(0))
        if k == "newton":
            out["norm"] = float(torch.linalg.norm(out["P_f"]))
    elif k == "strains":
        vals, F = E.assemble(_fluctuation(p, seed + 1), units)
        out = _named(p, vals, F)
        out["cases_f"] = F[1:, :p.n_free].flatten()
        out["cases_p"] = F[1:, p.n_free:].flatten()
    else:
        zero = np.zeros(p.n_nodes * p.dim)
        vals, F = E.assemble(zero, units if k == "request" else ())
        if k == "solve":
            b = E.t(np.random.default_rng(seed).uniform(-1.0, 1.0, c["rhs"] * p.n_free)).reshape(c["rhs"], -1)
            out = E.solve(vals[0], b).flatten()
        else:
            x = E.solve(vals[0], F[:, :p.n_free])
            C = np.zeros((len(units), len(units)))
            for j, e in enumerate(units):
                full = torch.cat([-x[j], torch.zeros(p.n_const, dtype=torch.float64, device=E.dev)])
                C[:, j] = E.average(full[E.dof.flatten()], e)
            out = {"x": x.flatten(), "C": C}
    p.close()
    return out
