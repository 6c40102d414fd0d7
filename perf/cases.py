"""The work a user of this library has it do, as measurable cases.

Each case is one call (or one short chain of calls) through the public Python
API over the C ABI, at the sizes of the named workloads and of ordinary
problems around them: whole fixed-source solves, the adjoint gradient, and the
single stages a host solver calls as shell operator and preconditioner (the
applies, the sweep, the element blocks, the DSA, the CG-SUPG operator).

Kinds:
    solve      TransportSolver.solve, then the scalar flux of the result
    gradient   DetectorResponse: forward solve, adjoint solve, both gradients
    apply      TransportOperator.mult             (L - S) x
    transpose  TransportOperator.mult_transpose   (L - S)^T x
    sweep      Sweep.apply                        L^{-1} q
    block      ElementBlockInverse.apply          element-block solves
    dsa        DSAPrecon.apply                    P D^{-1} R x, 30 inner iterations
    cg         the CG-SUPG operator's mult

The mesh of a size (and so its geometry tables and jitter) is the same for
every seed, as a program keeps one mesh for many cross sections; the cross
sections, sources and vectors come from the seed. `exact` takes the mesh's
geometry tables and the ordinates - the arrays a caller hands to the C ABI -
as given, and does everything else in torch in 64 bits.
"""
import functools
import math

import numpy as np
import torch

from ubolt_b200 import problem as P
from ubolt_b200 import transport as T

FACES = {"tri": 3, "quad": 4, "tet": 4, "hex": 6}
CELLS = {"tri": 2, "quad": 1, "tet": 6, "hex": 1}  # per box of the grid
DIM = {"tri": 2, "quad": 2, "tet": 3, "hex": 3}


def _case(name, kind, shape, n, order, sn, dtype="f64", **more):
    return dict({"name": name, "kind": kind, "shape": shape, "nx": n[0], "ny": n[1], "nz": n[2] if len(n) > 2 else 0,
                 "order": order, "sn": sn, "dtype": dtype, "reflect": False, "rtol": 0.0}, **more)


def listed():
    return [
        # The smallest whole solve: the structured 64 x 64 S4 problem as its
        # DG0 twin, to 1e-10 - launches, host round trips and latency
        _case("solve_quad64_dg0", "solve", "quad", (64, 64), 0, 4, rtol=1e-10),
        # The headline solve: 256 x 256 jittered quads as triangles, DG1, S8, to 1e-8
        _case("solve_tri256_dg1", "solve", "tri", (256, 256), 1, 8, rtol=1e-8),
        # FP32 inside FP64 refinement on jittered Kuhn tets in a scattering
        # medium, a smaller box of the combined 3D workload
        _case("solve_tet20_mixed", "solve", "tet", (20, 20, 20), 1, 8, "mixed", rtol=1e-10),
        # One evaluation of a detector response and its gradients, an
        # optimiser's step, on an ordinary ragged 2D mesh
        _case("gradient_tri_101x77", "gradient", "tri", (101, 77), 1, 6, rtol=1e-8),
        # The shell operator's multiply at the headline size
        _case("apply_tri256", "apply", "tri", (256, 256), 1, 8),
        # The FP32 multiply of a mixed solve on the 3D structured box: the largest vectors
        _case("apply_hex64_f32", "apply", "hex", (64, 64, 64), 1, 8, "f32"),
        # The adjoint's multiply on tets with two reflective (symmetry) sides
        _case("transpose_tet_23x21x19", "transpose", "tet", (23, 21, 19), 1, 6, reflect=True),
        # The streaming stage as a preconditioner call on a full right-hand side, a ragged mesh
        _case("sweep_tri_203x181", "sweep", "tri", (203, 181), 1, 8),
        # The same in FP32 on the 3D structured box
        _case("sweep_hex40_f32", "sweep", "hex", (40, 40, 40), 1, 8, "f32"),
        # The removal stage: the element-block solves on jittered quads
        _case("block_quad_301x257", "block", "quad", (301, 257), 1, 8),
        # The scattering stage: restriction, 30 inner iterations, prolongation
        _case("dsa_tri192", "dsa", "tri", (192, 192), 1, 8),
        # The vertex (CG-SUPG) backend's multiply
        _case("cg_quad256", "cg", "quad", (256, 256), 0, 8),
    ]


# Most rows (n_cells n_basis n_angles) a drawn case of a kind may have: no
# more work than the largest listed case
_MOST_ROWS = {"solve": 15.0e6, "gradient": 6.0e6, "apply": 42.0e6, "transpose": 20.0e6, "sweep": 20.0e6,
              "block": 30.0e6, "dsa": 18.0e6, "cg": 5.0e6}
_LEAST_ROWS = {"solve": 3.0e4, "gradient": 3.0e4, "apply": 3.0e4, "transpose": 3.0e4, "sweep": 3.0e4,
               "block": 3.0e4, "dsa": 3.0e4, "cg": 1.0e4}


def draw(rng):
    kind = rng.choice(["solve", "solve", "gradient", "apply", "apply", "transpose", "sweep", "sweep", "block", "dsa", "cg"])
    shape = rng.choice(["tri", "tri", "quad", "tet", "hex"])
    order = 1 if kind in ("dsa", "gradient") else rng.choice([0, 1, 1, 1])
    if kind == "cg":
        order = 0
    dim = DIM[shape]
    sn = rng.choice([2, 4, 6, 8, 8, 10, 12] if dim == 2 else [2, 4, 6, 8, 8])
    dtype = {"solve": rng.choice(["f64", "f64", "mixed"]), "gradient": "f64", "dsa": "f64"}.get(
        kind, rng.choice(["f64", "f64", "f32"]))
    na = sn * (sn + 2) // 2 if dim == 2 else sn * (sn + 2)
    nb = dim + 1 if order else 1
    lo, hi = _LEAST_ROWS[kind], _MOST_ROWS[kind]
    rows = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    boxes = max(8.0, rows / (nb * na * CELLS[shape]))
    # A box of about that many cells, its sides within a third of each other
    n = [max(2, round(boxes ** (1.0 / dim) * rng.uniform(0.75, 1.3))) for _ in range(dim)]
    limit = 66 if dim == 3 else 600
    n = [min(limit, k) for k in n]
    while (n[0] * n[1] * (n[2] if dim == 3 else 1)) * CELLS[shape] * nb * na > hi:
        n[n.index(max(n))] -= 1
    case = _case("", kind, shape, n, order, sn, dtype)
    del case["name"]
    if kind in ("apply", "transpose"):
        case["reflect"] = rng.random() < 0.25
    if kind in ("solve", "gradient"):
        case["rtol"] = 1e-10 if dtype == "mixed" else rng.choice([1e-8, 1e-10])
    return case


# ~~~ Meshes, cross sections, vectors


@functools.lru_cache(maxsize=2)
def _geometry(shape, nx, ny, nz, order, reflect, cg):
    rng = np.random.default_rng(nx * 7919 + ny * 104729 + nz)
    if shape == "tri":
        mesh = P.box_tris(nx, ny, jitter=0.2, rng=rng)
    elif shape == "quad":
        mesh = P.box_quads(nx, ny, jitter=0.2 if order or cg else 0.0, rng=rng)
    elif shape == "tet":
        mesh = P.box_tets(nx, ny, nz, jitter=0.2, rng=rng)
    else:
        mesh = P.box_hexes(nx, ny, nz)
    if cg:
        return P.build_cg_geometry(mesh)
    bc = np.zeros(2 * DIM[shape], dtype=np.int32)
    if reflect:
        bc[0] = bc[2] = 1
    return P.build_geometry(mesh, order, side_bc=bc)


def _setting(case):
    g = _geometry(case["shape"], case["nx"], case["ny"], case["nz"], case["order"], case["reflect"],
                  case["kind"] == "cg")
    return g, P.lqn(DIM[case["shape"]], case["sn"])


def _inputs(case, seed, g, q):
    """Cross sections, source and vectors from the seed, on the GPU, FP64."""
    r = torch.Generator().manual_seed(int(seed) * 1000003 + 12345)
    nc = g.n_cells
    unif = lambda lo, hi: lo + (hi - lo) * torch.rand(nc, generator=r, dtype=torch.float64)
    if case["shape"] == "hex":
        # Constant over blocks, 0.1 to 10 mean free paths, as a material map has them
        c = torch.from_numpy(np.ascontiguousarray(g.centroid.reshape(-1, 3)))
        blk = (c * 8).long().clamp(max=7)
        bid = (blk[:, 2] * 8 + blk[:, 1]) * 8 + blk[:, 0]
        st = (10.0 ** (2.0 * torch.rand(512, generator=r, dtype=torch.float64) - 1.0))[bid]
        ratio = (0.5 + 0.4 * torch.rand(512, generator=r, dtype=torch.float64))[bid]
    else:
        spread, lo, hi = (1.0, 0.5, 0.999) if case["shape"] == "tet" else (0.5, 0.3, 0.99)
        st = torch.exp(spread * torch.randn(nc, generator=r, dtype=torch.float64))
        ratio = unif(lo, hi)
    src = (unif(0.0, 1.0) < 0.3).double()
    det = (unif(0.0, 1.0) < 0.05).double()
    dev = torch.device("cuda")
    rows = (g.n_cells * getattr(g, "n_basis", 1) if case["kind"] != "cg" else g.n_vertices) * q.n_angles
    out = {"st": st.to(dev), "ss": (ratio * st).to(dev), "src": src.to(dev), "det": det.to(dev)}
    if case["kind"] not in ("solve", "gradient"):
        gd = torch.Generator(device=dev).manual_seed(int(seed) * 1000003 + 54321)
        x = torch.randn(rows, generator=gd, dtype=torch.float64, device=dev)
        out["x"] = x.float() if case["dtype"] == "f32" else x
    return out


def prepare(case, seed):
    g, q = _setting(case)
    d = _inputs(case, seed, g, q)
    ctx = T.Context(g, q)
    kind = case["kind"]
    s = {"kind": kind, "ctx": ctx, **d}
    if kind == "gradient":
        # The response object is what an optimiser keeps; the cross sections change per evaluation
        ctx.set_group(d["st"], d["ss"])
        s["model"] = T.DetectorResponse(ctx, d["src"], d["det"], rtol=case["rtol"], precision="fp64", pc="sweep")
        return s
    ctx.set_group(d["st"], d["ss"])
    if kind == "solve":
        b = ctx.vector(fill=0.0)
        T.GroupTransfer(ctx, [[d["ss"]]], [d["src"]]).add_external(0, b)
        s["b"], s["psi"] = b, ctx.vector()
        s["solver"] = T.TransportSolver(ctx, rtol=case["rtol"], pc="sweep",
                                        precision="mixed" if case["dtype"] == "mixed" else "fp64")
    elif kind == "sweep":
        s["op"] = T.Sweep(ctx)
        s["y"] = torch.empty_like(d["x"])
    elif kind == "dsa":
        s["op"] = T.DSAPrecon(ctx)
        s["op"].set_group()
        s["y"] = torch.empty_like(d["x"])
    else:
        s["op"] = T.ElementBlockInverse(ctx) if kind == "block" else T.TransportOperator(ctx)
        s["y"] = torch.empty_like(d["x"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "solve":
        x, _ = s["solver"].solve(s["b"], s["psi"])
        return {"psi": x, "phi": T.angular_integral(s["ctx"], x)}
    if kind == "gradient":
        st, ss = s["st"].detach().requires_grad_(), s["ss"].detach().requires_grad_()
        J = s["model"](st, ss)
        gt, gs = torch.autograd.grad(J, (st, ss))
        return {"J": J.detach(), "grad_sigma_t": gt, "grad_sigma_s": gs}
    if kind == "transpose":
        return s["op"].mult_transpose(s["x"], s["y"])
    if kind in ("apply", "cg"):
        return s["op"].mult(s["x"], s["y"])
    return s["op"].apply(s["x"], s["y"])


def work(case):
    """Vectors in and out and the per-cell cross sections, once each; the
    multiply-adds of the streaming blocks, two flops each."""
    dim, shape = DIM[case["shape"]], case["shape"]
    boxes = case["nx"] * case["ny"] * (case["nz"] if dim == 3 else 1)
    nc = boxes * CELLS[shape]
    nb = dim + 1 if case["order"] else 1
    na = case["sn"] * (case["sn"] + 2) // (2 if dim == 2 else 1)
    el = 4 if case["dtype"] == "f32" else 8
    F = FACES[shape]
    if case["kind"] == "cg":
        nv = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1 if dim == 3 else 1)
        verts = {"tri": 3, "quad": 4, "tet": 4, "hex": 8}[shape]
        return {"bytes": 2 * nv * na * el + 2 * nc * 8, "flops": 4.0 * nc * verts * verts * na}
    rows = nc * nb * na
    flops = 2.0 * rows * nb * (F + 1)
    if case["kind"] == "solve":
        return {"bytes": 2 * rows * 8 + nc * nb * 8 + 2 * nc * 8, "flops": 2 * flops}
    if case["kind"] == "gradient":
        return {"bytes": 4 * rows * 8 + 6 * nc * 8, "flops": 4 * flops}
    return {"bytes": 2 * rows * el + 2 * nc * el, "flops": flops}


# ~~~ The same in 64 bits with torch alone


class _Dg:
    """The DG operator on the geometry tables, dense over (cell, ordinate)."""

    def __init__(self, g, q, st, ss, dev):
        t = lambda a, *shape: torch.from_numpy(np.ascontiguousarray(a)).to(dev).reshape(*shape)
        self.nc, self.nb, self.F, self.A = g.n_cells, g.n_basis, g.faces_per_cell, q.n_angles
        nc, nb, F = self.nc, self.nb, self.F
        self.vol = t(g.volume, nc)
        self.nA, self.nbr = t(g.face_nA, nc, F, 3), t(g.face_neighbour, nc, F).long()
        self.side, self.bc = t(g.face_side, nc, F).long(), t(g.face_bc, nc, F)
        if nb > 1:
            self.fown, self.fup = t(g.face_own, nc, F, nb, nb), t(g.face_up, nc, F, nb, nb)
            self.grad = t(g.basis_grad, nc, nb, 3)
        else:
            self.fown = self.fup = (1.0 / self.vol)[:, None, None, None].expand(nc, F, 1, 1)
            self.grad = torch.zeros(nc, 1, 3, dtype=torch.float64, device=dev)
        self.om, self.w = t(q.omega, self.A, 3), t(q.w, self.A)
        self.refl, self.W = t(q.reflect, 3, self.A).long(), q.sum_weights
        self.opp = t(q.opposite(), self.A).long()
        self.st, self.ss, self.dev = st.to(dev), ss.to(dev), dev

    def apply(self, x, scatter=True):
        nc, nb, A = self.nc, self.nb, self.A
        x = x.reshape(nc, nb, A)
        y = self.st[:, None, None] * x
        if nb > 1:
            y[:, 1:] = y[:, 1:] - (self.grad[:, 1:] @ self.om.T) * x[:, :1]
        for f in range(self.F):
            s = self.nA[:, f] @ self.om.T
            y = y + s.clamp(min=0.0)[:, None, :] * (self.fown[:, f] @ x)
            inner = self.nbr[:, f] >= 0
            up = torch.where(inner[:, None, None], x[self.nbr[:, f].clamp(min=0)], 0.0)
            mirror = ~inner & (self.bc[:, f] == 1)
            if bool(mirror.any()):
                ar = self.refl[(self.side[:, f].clamp(min=0) // 2)]
                up = torch.where(mirror[:, None, None], torch.gather(x, 2, ar[:, None, :].clamp(min=0).expand(-1, nb, -1)), up)
            y = y + s.clamp(max=0.0)[:, None, :] * (self.fup[:, f] @ up)
        if scatter:
            y = y - (self.ss / self.W)[:, None, None] * (x @ self.w)[:, :, None]
        return y.reshape(-1)

    def blocks(self):
        nc, nb, A = self.nc, self.nb, self.A
        B = torch.zeros(nc, A, nb, nb, dtype=torch.float64, device=self.dev)
        for f in range(self.F):
            s = (self.nA[:, f] @ self.om.T).clamp(min=0.0)
            B += s[:, :, None, None] * self.fown[:, f][:, None]
        if nb > 1:
            B[:, :, 1:, 0] -= (self.grad[:, 1:] @ self.om.T).transpose(1, 2)
        return B + self.st[:, None, None, None] * torch.eye(nb, dtype=torch.float64, device=self.dev)

    def plan(self):
        """Upwind levels over all ordinates at once: flat (cell, ordinate) indices per level."""
        nc, F, A = self.nc, self.F, self.A
        s = torch.stack([self.nA[:, f] @ self.om.T for f in range(F)], 1)  # (nc, F, A)
        up = (s < 0) & (self.nbr >= 0)[:, :, None]
        # The slot of the neighbour that faces back
        back = torch.full((nc, F), -1, dtype=torch.long, device=self.dev)
        cells = torch.arange(nc, device=self.dev)
        for f in range(F):
            for h in range(F):
                n = self.nbr[:, f]
                hit = (n >= 0) & (self.nbr[n.clamp(min=0), h] == cells)
                back[:, f] = torch.where(hit, h, back[:, f])
        indeg = up.sum(1).reshape(-1).int()
        front = torch.nonzero(indeg == 0).reshape(-1)
        self.levels, done = [], 0
        while front.numel():
            self.levels.append(front)
            done += front.numel()
            c, a = front // A, front % A
            n, h = self.nbr[c], back[c]
            reads = (n >= 0) & up[n.clamp(min=0), h.clamp(min=0), a[:, None]]
            down = (n * A + a[:, None])[reads]
            indeg.index_add_(0, down, torch.full((down.numel(),), -1, dtype=torch.int32, device=self.dev))
            down = torch.unique(down)
            front = down[indeg[down] == 0]
        self.acyclic = done == nc * A
        self.s = s
        self.inv = torch.linalg.inv(self.blocks())  # (nc, A, nb, nb)

    def sweep(self, q):
        nc, nb, F, A = self.nc, self.nb, self.F, self.A
        q = q.reshape(nc, nb, A)
        psi = torch.zeros(nc, A, nb, dtype=torch.float64, device=self.dev)
        for idx in self.levels:
            c, a = idx // A, idx % A
            r = q[c, :, a]
            n = self.nbr[c]
            sm = self.s[c, :, a].clamp(max=0.0) * (n >= 0)
            xu = psi[n.clamp(min=0), a[:, None]]  # (m, F, nb)
            r = r - (sm[:, :, None] * (self.fup[c] @ xu[..., None])[..., 0]).sum(1)
            psi[c, a] = (self.inv[c, a] @ r[..., None])[..., 0]
        return psi.transpose(1, 2).reshape(-1)

    def sweep_t(self, q):
        """L^{-T} q = V P L^{-1} P V^{-1} q, P the swap of opposite ordinates."""
        v = self.vol[:, None, None]
        z = (q.reshape(self.nc, self.nb, self.A) / v)[:, :, self.opp]
        z = self.sweep(z.reshape(-1)).reshape(self.nc, self.nb, self.A)
        return (z[:, :, self.opp] * v).reshape(-1)

    def solve(self, b, transpose=False):
        """(L - S) x = b (or its transpose) by GMRES on the scattering moment:
        m = M L^{-1}(b + E m), E m the source of a moment."""
        nc, nb, A = self.nc, self.nb, self.A
        sg = (self.ss / self.W)[:, None]
        if transpose:
            moment = lambda x: (sg * x.reshape(nc, nb, A).sum(-1)).reshape(-1)
            spread = lambda m: (m[:, None] * self.w[None, :]).reshape(-1)
            inv = self.sweep_t
        else:
            moment = lambda x: (sg * (x.reshape(nc, nb, A) @ self.w)).reshape(-1)
            spread = lambda m: m[:, None].expand(-1, A).reshape(-1)
            inv = self.sweep
        r0 = moment(inv(b))
        beta = torch.linalg.norm(r0)
        if float(beta) == 0.0:
            return inv(b)
        V, H, m = [r0 / beta], np.zeros((61, 60)), None
        for j in range(60):
            w = V[j] - moment(inv(spread(V[j])))
            for _ in range(2):
                for i, v in enumerate(V):
                    h = torch.dot(v, w)
                    H[i, j] += float(h)
                    w = w - h * v
            H[j + 1, j] = float(torch.linalg.norm(w))
            e = np.zeros(j + 2)
            e[0] = float(beta)
            y = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)[0]
            m = sum(float(y[i]) * V[i] for i in range(j + 1))
            if np.linalg.norm(H[:j + 2, :j + 1] @ y - e) < 1e-14 * float(beta) or H[j + 1, j] == 0.0:
                break
            V.append(w / H[j + 1, j])
        return inv(b + spread(m))


def _mip_apply(g, q, st, ss, x, dev, its=30, penalty=4.0):
    """P D^{-1} R x with the interior-penalty D of DG1 and `its` block-Jacobi PCG iterations."""
    t = lambda a, *shape: torch.from_numpy(np.ascontiguousarray(a)).to(dev).reshape(*shape)
    nc, nb, F, A = g.n_cells, g.n_basis, g.faces_per_cell, q.n_angles
    vol, nbr, bc = t(g.volume, nc), t(g.face_neighbour, nc, F).long(), t(g.face_bc, nc, F)
    nA, dist = t(g.face_nA, nc, F, 3), t(g.face_distance, nc, F, 2)
    fo, fu = t(g.face_own, nc, F, nb, nb), t(g.face_up, nc, F, nb, nb)
    gr, gn_ = t(g.basis_grad, nc, nb, 3), t(g.face_neighbour_grad, nc, F, nb, 3)
    w = t(q.w, A)
    D = 1.0 / (3.0 * st)
    area = torch.linalg.norm(nA, dim=-1)
    nrm = nA / area[..., None]
    own = vol[:, None, None] * (D[:, None, None] * (gr @ gr.transpose(1, 2)) +
                                (st - ss)[:, None, None] * torch.eye(nb, dtype=torch.float64, device=dev))
    off = torch.zeros(nc, F, nb, nb, dtype=torch.float64, device=dev)
    for f in range(F):
        n = nbr[:, f]
        inner, vac = n >= 0, (n < 0) & (bc[:, f] == 0)
        sc = vol * area[:, f]
        gc, gn = (gr @ nrm[:, f, :, None])[..., 0], (gn_[:, f] @ nrm[:, f, :, None])[..., 0]
        Dn = D[n.clamp(min=0)]
        hc, hn = 2.0 * dist[:, f, 0], 2.0 * dist[:, f, 1]
        ki = (0.5 * penalty * (D / hc + Dn / torch.where(inner, hn, 1.0))).clamp(min=0.25)
        kv = (penalty * D / hc).clamp(min=0.25)
        mi = sc[:, None] * fo[:, f, :, 0]
        half = (0.5 * D)[:, None, None]
        a = (torch.where(inner, ki, kv) * sc)[:, None, None] * fo[:, f] \
            - half * gc[:, None, :] * mi[:, :, None] - half * gc[:, :, None] * (sc[:, None] * fo[:, f, 0])[:, None, :]
        own = own + torch.where((inner | vac)[:, None, None], a, 0.0)
        o = -(ki * sc)[:, None, None] * fu[:, f] - (0.5 * Dn)[:, None, None] * gn[:, None, :] * mi[:, :, None] \
            + half * gc[:, :, None] * (sc[:, None] * fu[:, f, 0])[:, None, :]
        off[:, f] = torch.where(inner[:, None, None], o, 0.0)
    jinv = torch.linalg.inv(own)
    mul = lambda M, u: (M @ u[..., None])[..., 0]

    def spmv(u):
        v = mul(own, u)
        for f in range(F):
            v = v + mul(off[:, f], u[nbr[:, f].clamp(min=0)])
        return v

    r = vol[:, None] * (x.reshape(nc, nb, A) @ w)
    u = torch.zeros_like(r)
    z = mul(jinv, r)
    p, rho = z, (r * z).sum()
    for _ in range(its):
        v = spmv(p)
        al = rho / (p * v).sum()
        u, r = u + al * p, r - al * v
        z = mul(jinv, r)
        new = (r * z).sum()
        p, rho = z + (new / rho) * p, new
    return (u / q.sum_weights)[..., None].expand(-1, -1, A).reshape(-1)


def _cg_apply(g, q, st, ss, x, dev, zeta=0.5):
    """The SUPG operator, element by element: gather, multiply, add to the vertices."""
    t = lambda a, *shape: torch.from_numpy(np.ascontiguousarray(a)).to(dev).reshape(*shape)
    ne, nv, nx, A, dim = g.n_elements, g.n_element_vertices, g.n_vertices, q.n_angles, g.dim
    ev = t(g.elem_vertex, ne, nv).long()
    M, G, K = t(g.mass, ne, nv, nv), t(g.grad, ne, nv, nv, 3), t(g.stiff, ne, nv, nv, 3, 3)
    cg, lumped = t(g.centre_grad, ne, nv, 3), t(g.lumped_mass, nx)
    om, w = t(q.omega, A, 3).clone(), t(q.w, A)
    om[:, dim:] = 0.0
    x = x.reshape(nx, A)
    phi = x @ w
    y = torch.zeros(nx, A, dtype=torch.float64, device=dev)
    for a in range(A):
        thin = 2.0 / (zeta * (cg @ om[a]).abs().sum(1))
        tau = torch.where(st > 0, torch.minimum(1.0 / st, thin), thin)[:, None, None]
        og = G @ om[a]
        wt = M + tau * og.transpose(1, 2)
        kk = torch.einsum("eijkl,k,l->eij", K, om[a], om[a])
        coef = og + tau * kk + st[:, None, None] * wt
        r = (coef @ x[ev, a][..., None])[..., 0] - (ss / q.sum_weights)[:, None] * (wt @ phi[ev][..., None])[..., 0]
        y[:, a].index_add_(0, ev.reshape(-1), r.reshape(-1))
    y = y / lumped[:, None]
    # The weak inflow faces (vacuum sides)
    off = t(g.bface_offset, nx + 1).long()
    vtx = torch.repeat_interleave(torch.arange(nx, device=dev), off[1:] - off[:-1])
    s = (t(g.bface_nA, -1, 3) @ om.T).clamp(max=0.0)
    return y.index_add(0, vtx, -s * t(g.bface_mass, -1)[:, None] * x[vtx]).reshape(-1)


def exact(case, seed):
    g, q = _setting(case)
    d = _inputs(case, seed, g, q)
    dev = torch.device("cuda")
    st, ss, kind = d["st"], d["ss"], case["kind"]
    x = d["x"].double() if "x" in d else None
    if kind == "cg":
        return _cg_apply(g, q, st, ss, x, dev)
    if kind == "dsa":
        return _mip_apply(g, q, st, ss, x, dev)
    op = _Dg(g, q, st, ss, dev)
    if kind == "apply":
        return op.apply(x)
    if kind == "transpose":
        x = x.reshape(op.nc, op.nb, op.A)
        z = torch.zeros_like(x).reshape(-1).requires_grad_()
        return torch.autograd.grad(op.apply(z), z, x.reshape(-1))[0]
    if kind == "block":
        xb = x.reshape(op.nc, op.nb, op.A).transpose(1, 2)
        y = torch.linalg.solve(op.blocks(), xb[..., None])[..., 0]
        return y.transpose(1, 2).reshape(-1)
    op.plan()
    if not op.acyclic:
        return None
    if kind == "sweep":
        return op.sweep(x)
    b = torch.zeros(op.nc, op.nb, op.A, dtype=torch.float64, device=dev)
    b[:, 0] = (d["src"] / q.sum_weights)[:, None]
    psi = op.solve(b.reshape(-1))
    if kind == "solve":
        return {"psi": psi, "phi": (psi.reshape(-1, op.A) @ op.w)}
    r = torch.zeros(op.nc, op.nb, op.A, dtype=torch.float64, device=dev)
    r[:, 0] = (d["det"] * op.vol)[:, None] * op.w
    lam = op.solve(r.reshape(-1), transpose=True).reshape(op.nc, op.nb, op.A)
    p = psi.reshape(op.nc, op.nb, op.A)
    return {"J": (r * p).sum(), "grad_sigma_t": -(lam * p).sum((1, 2)),
            "grad_sigma_s": (lam.sum(-1) * (p @ op.w)).sum(-1) / q.sum_weights}
