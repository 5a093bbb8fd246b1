"""Timed cases of the solver: what a program that uses the library has it do, over the sizes, meshes,
equations, precisions and entry points that it offers.

kind "solve"    one resident solve: restart from a state, advance one monitor interval, read the
                solution back (the driver's loop between two outputs)
kind "coupled"  a host program that owns the state: it hands the state over, advances one iteration
                and takes the state back, several times in a row
kind "batch"    many independent solves on one GPU: admit them, advance them together, read the
                residual norms and every solution, retire them (one round of a sweep or a server)
kind "noalloc"  one first-order residual on device arrays the caller owns
Meshes come from the package's generators; ``exact`` restates the method in 64 bits with torch alone.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from __graft_entry__ import load_package

PKG = load_package()
BC = {"FREESTREAM": -1, "SLIP_WALL": -2, "EXTRAPOLATION": -3, "NO_SLIP_WALL": -4}


# ------------------------------------------------------------------------------------------ cases
def _solve(name, mesh, cells, eqn, precision, iterations, order=1, limiter="SQUEEZE", dt="LOCAL", cfl=0.5,
           mach=0.5, reynolds=5000.0, kind="solve", solves=1):
    return dict(name=name, kind=kind, mesh=mesh, cells=cells, eqn=eqn, precision=precision, iterations=iterations,
                order=order, limiter=limiter, dt=dt, cfl=cfl, mach=mach, reynolds=reynolds, solves=solves)


def listed():
    return [
        # the smallest call: a 32 x 16 channel, as a smoke check or a first try of an input file runs it
        _solve("tiny quads fp64", "quads", 512, "EULER", "fp64", 50, dt="GLOBAL", cfl=0.8),
        # the reference program's own kind of case: 128 x 64 bump channel, one global time step
        _solve("channel quads fp64", "quads", 8192, "EULER", "fp64", 50, dt="GLOBAL", cfl=0.8),
        # the same size on polygons, viscous, in single precision: an airfoil- or cylinder-sized solve
        _solve("cylinder 12k fp32", "cylinder", 12000, "NS", "fp32", 50, mach=0.2, reynolds=100.0),
        # an ordinary engineering mesh, inviscid, single precision
        _solve("bump 50k fp32", "bump", 50000, "EULER", "fp32", 50, dt="GLOBAL", cfl=0.8, mach=0.7),
        # an ordinary engineering mesh, viscous, double precision
        _solve("bump 50k ns fp64", "bump", 50000, "NS", "fp64", 20, mach=0.4),
        # first order on a large mesh, as the precision study and start-up runs use it
        _solve("first order 300k fp32", "bump", 300000, "EULER", "fp32", 50, order=0, limiter="NONE", cfl=0.8,
               mach=0.7),
        # the headline workload (viscous cylinder, about a million polygonal cells) in both precisions
        _solve("cylinder 1M fp64", "cylinder", 1000000, "NS", "fp64", 5, mach=0.2, reynolds=100.0),
        _solve("cylinder 1M fp32", "cylinder", 1000000, "NS", "fp32", 50, mach=0.2, reynolds=100.0),
        # a host code that keeps the state itself, as the reference's main() does
        _solve("coupled 100k fp64", "cylinder", 100000, "NS", "fp64", 5, mach=0.2, reynolds=100.0, kind="coupled"),
        # a parameter sweep in single precision, and a smaller one in double
        _solve("batch 96 fp32", "mixed", 2400000, "MIXED", "fp32", 100, kind="batch", solves=96),
        _solve("batch 12 fp64", "mixed", 60000, "MIXED", "fp64", 20, kind="batch", solves=12),
        # the residual for a caller that cannot allocate, near that entry's face limit
        _solve("noalloc 86k", "bump", 86000, "EULER", "fp64", 1, order=0, limiter="NONE", mach=0.6, kind="noalloc"),
    ]


def draw(rng):
    """One more case: sizes log-uniform over the range, the options mixed as users mix them."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve"] * 6 + ["coupled", "batch", "batch", "noalloc"])
    if kind == "noalloc":
        return {k: v for k, v in _solve("", rng.choice(["bump", "quads"]), size(120, 86000), rng.choice(["EULER", "NS"]),
                                        "fp64", 1, order=0, limiter="NONE", mach=rng.uniform(0.3, 0.7),
                                        kind="noalloc").items() if k != "name"}
    precision = rng.choice(["fp32", "fp64"])
    if kind == "batch":
        n = rng.choice([3, 7, 16, 24, 40, 64])
        top = 1500000 if precision == "fp32" else 250000
        c = _solve("", "mixed", min(top, n * size(600, 40000)), "MIXED", precision,
                   rng.randint(30, 100) if precision == "fp32" else rng.randint(5, 20), kind="batch", solves=n)
    else:
        mesh = rng.choice(["quads", "cylinder", "bump", "bump"])
        eqn = rng.choice(["EULER", "NS"])
        order = rng.choice([0, 1, 1, 1, 1])
        limiter = "NONE" if order == 0 else rng.choice(["SQUEEZE", "SQUEEZE", "SQUEEZE", "NONE"])
        lo = 3000 if mesh == "cylinder" else 200
        cells = size(lo, 400000)
        its = rng.randint(2, 5) if kind == "coupled" else rng.randint(10, 60)
        if precision == "fp64":
            its = max(2, min(its, 3000000 // cells))
        ns = eqn == "NS"
        c = _solve("", mesh, cells, eqn, precision, its, order=order, limiter=limiter,
                   dt=rng.choice(["GLOBAL", "LOCAL"]), cfl=0.5 if ns or mesh == "cylinder" else rng.uniform(0.5, 0.8),
                   mach=0.2 if mesh == "cylinder" else rng.uniform(0.3, 0.7),
                   reynolds=rng.uniform(80, 200) if mesh == "cylinder" else rng.uniform(3e3, 1e4), kind=kind)
    return {k: v for k, v in c.items() if k != "name"}


# ----------------------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=16)
def _grid(mesh, cells, seed):
    mg = PKG.meshgen
    if mesh == "quads":
        ny = max(4, int(round(math.sqrt(cells / 2.0))))
        return mg.channel_bump_quads(max(4, int(round(cells / ny))), ny)
    if mesh == "bump":
        return mg.voronoi_bump_channel(cells, seed=seed)
    if cells >= 250000:   # the benchmark's box
        return mg.voronoi_cylinder(cells, seed=seed)
    # smaller boxes for smaller meshes: the generator's far-field spacing sets a least cell count
    return mg.voronoi_cylinder(cells, seed=seed, box=(6.0, 3.0), h_wall=0.01 if cells < 40000 else 0.004,
                               h_far=0.25 if cells < 8000 else 0.08)


def _options(case):
    """The input-file options of a solve."""
    mg = PKG.meshgen
    U = mg.mach_speed(case["mach"])
    ns = case["eqn"] == "NS"
    wall = "NO_SLIP_WALL" if ns else "SLIP_WALL"
    return dict(mg.DEFAULT_CASE, eqn=case["eqn"], solution_poly_order=case["order"], limiter=case["limiter"],
                time_step_type=case["dt"], CFL=case["cfl"], u=U * math.cos(0.02), v=U * math.sin(0.02),
                mu=1.225 * U / case["reynolds"] if ns else 0.0, Pr=0.72, BC1=wall, BC2="FREESTREAM")


def _state(case, opt, grid, seed):
    """A developing flow to restart from: the freestream with smooth waves of a few percent and a
    weak pressure front, 4N doubles in the file's numbering."""
    rng = np.random.default_rng(seed)
    x = np.empty(grid.num_cells)
    y = np.empty(grid.num_cells)
    inter = grid.fc2 > 0
    cells = np.concatenate([grid.fc1, grid.fc2[inter]]) - 1
    count = np.bincount(cells, minlength=grid.num_cells)
    for out, p in ((x, grid.x), (y, grid.y)):
        mid = 0.5 * (p[grid.fp1 - 1] + p[grid.fp2 - 1])
        out[:] = np.bincount(cells, weights=np.concatenate([mid, mid[inter]]), minlength=grid.num_cells) / count
    span = max(x.max() - x.min(), y.max() - y.min())
    x, y = (x - x.min()) / span, (y - y.min()) / span

    def wave():
        w = np.zeros_like(x)
        for _ in range(3):
            kx, ky, ph = rng.uniform(2, 14), rng.uniform(2, 14), rng.uniform(0, 2 * math.pi)
            w += np.sin(kx * x + ky * y + ph) / 3
        return w

    front = np.tanh((x - rng.uniform(0.3, 0.7)) / 0.02)
    rho = opt["rho"] * (1 + 0.03 * wave() - 0.015 * front)
    P = opt["P"] * (1 + 0.04 * wave() - 0.02 * front)
    U = math.hypot(opt["u"], opt["v"])
    u = opt["u"] + 0.05 * U * wave()
    v = opt["v"] + 0.05 * U * wave()
    E = P / (opt["gamma"] - 1) + 0.5 * rho * (u * u + v * v)
    return np.concatenate([rho, rho * u, rho * v, E])


def _batch_solves(case, seed):
    """(mesh key, case) of every solve of a batch: a few meshes, flow conditions drawn per solve."""
    rng = np.random.default_rng(seed)
    shapes = np.random.default_rng(case["cells"] + case["solves"])   # the meshes belong to the case
    n = case["solves"]
    kinds = min(n, 6)
    share = np.exp(shapes.uniform(-1.2, 1.2, kinds))
    share = share / share.sum() * case["cells"] / n * kinds
    out = []
    for i in range(n):
        k = i % kinds
        mesh = "quads" if k == 2 else "bump"
        ns = mesh == "bump" and k % 2 == 1
        c = dict(case, mesh=mesh, cells=max(60, int(share[k])), eqn="NS" if ns else "EULER", order=1, limiter="SQUEEZE",
                 dt="GLOBAL" if k == 4 else "LOCAL", cfl=0.5 if ns else 0.8, mach=float(rng.uniform(0.3, 0.7)),
                 reynolds=float(rng.uniform(3e3, 1e4)))
        out.append(((mesh, c["cells"], k), c))
    return out


class _NoallocMesh(ctypes.Structure):
    _fields_ = [("num_cells", ctypes.c_int), ("num_faces", ctypes.c_int)] + [
        (k, ctypes.c_void_p) for k in ("face_cell1", "face_cell2", "face_nx", "face_ny", "face_area",
                                       "cell_face_offsets", "cell_faces", "cell_vol")]


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True)


def prepare(case, seed):
    precision = PKG.FP64 if case["precision"] == "fp64" else PKG.FP32
    if case["kind"] == "batch":
        solves = _batch_solves(case, seed)
        meshes, n_cells, n_faces = {}, 0, 0
        for key, c in solves:
            g = _grid(*key)
            if key not in meshes:
                meshes[key] = PKG.HostMesh(g, PKG.case_from_dict(_options(c)))
            n_cells += g.num_cells
            n_faces += g.num_faces
        batch = PKG.Batch(n_cells + 64 * len(solves), n_faces + 64 * len(solves), len(solves), precision=precision)
        return dict(kind="batch", batch=batch, precision=precision, iterations=case["iterations"],
                    solves=[(meshes[key], PKG.case_from_dict(_options(c))) for key, c in solves])
    grid = _grid(case["mesh"], case["cells"], 1)
    opt = _options(case)
    q = _state(case, opt, grid, seed)
    cs = PKG.case_from_dict(opt)
    if case["kind"] == "noalloc":
        hm = PKG.HostMesh(grid, cs)
        nf, nc = grid.num_faces, grid.num_cells
        fc1 = grid.fc1.astype(np.int64) - 1
        fc2 = np.where(grid.fc2 > 0, grid.fc2 - 1, np.where(grid.fc2 == 0, BC[opt["BC1"]], BC[opt["BC2"]]))
        f = np.arange(nf)
        inter = fc2 >= 0
        cells = np.concatenate([fc1, fc2[inter]])
        ent = np.concatenate([f << 1, (f[inter] << 1) | 1])
        order = np.lexsort((ent >> 1, cells))
        off = np.concatenate([[0], np.cumsum(np.bincount(cells, minlength=nc))])
        dev = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, dtype=t)).cuda()  # noqa: E731
        arrays = [dev(fc1, np.int32), dev(fc2, np.int32)] + [dev(hm.geom(k), np.float64) for k in ("nx", "ny", "area")]
        arrays += [dev(off, np.int32), dev(ent[order], np.int32), dev(hm.geom("vol"), np.float64)]
        fn = PKG.library().fv2d_residual_noalloc
        fn.restype = ctypes.c_int
        fn.argtypes = [ctypes.POINTER(_NoallocMesh), ctypes.POINTER(PKG.Case), ctypes.c_void_p, ctypes.c_void_p,
                       ctypes.c_void_p]
        return dict(kind="noalloc", fn=fn, mesh=_NoallocMesh(nc, nf, *[a.data_ptr() for a in arrays]), arrays=arrays,
                    case=cs, q=dev(q, np.float64), r=torch.empty(4 * nc, dtype=torch.float64, device="cuda"))
    host = _pinned(q.size)
    host.copy_(torch.from_numpy(q))
    return dict(kind=case["kind"], solver=PKG.Solver(grid, cs, precision=precision), precision=precision,
                iterations=case["iterations"], q=host, out=_pinned(q.size))


def run(state):
    kind = state["kind"]
    if kind == "noalloc":
        stream = torch.cuda.current_stream().cuda_stream
        rc = state["fn"](ctypes.byref(state["mesh"]), ctypes.byref(state["case"]), state["q"].data_ptr(),
                         state["r"].data_ptr(), stream)
        if rc:
            raise RuntimeError(f"fv2d_residual_noalloc: {rc}")
        return state["r"]
    if kind == "batch":
        b = state["batch"]
        ids = [b.add_mesh(m, cs) for m, cs in state["solves"]]
        b.step(state["iterations"])
        norms = b.norms()
        q = np.concatenate([b.get_state(i) for i in ids])
        r = np.stack([norms[i][0] for i in ids])
        for i in ids:
            b.remove(i)
        if state["precision"] == PKG.FP64:
            return q, r
        return torch.from_numpy(q).cuda().float()   # single precision: the solutions in that precision
    s, out = state["solver"], state["out"].numpy()
    s.set_state(state["q"].numpy())
    if kind == "coupled":
        for k in range(state["iterations"]):
            if k:
                s.load_state(out)
            s.step(1)
            s.get_state(out)
    else:
        s.step(state["iterations"])
        s.get_state(out)
    if state["precision"] == PKG.FP64:
        return state["out"], s.residual_norm()
    s.residual_norm()   # the monitor line
    return state["out"].cuda().float()   # handed on in the precision that it was computed in


# ------------------------------------------------------------------------------------------- work
def work(case):
    """Of one pass: a stage reads the state, the face geometry (normal, area, two offsets, two ids)
    and the cell geometry, and writes the state; a pass moves the state in and out once.  Arithmetic:
    per face and per cell, counted from the method's formulas."""
    s = 8 if case["precision"] == "fp64" else 4
    n, faces = case["cells"], (2.1 if case["mesh"] == "quads" else 3.0) * case["cells"]
    if case["kind"] == "noalloc":
        return {"bytes": 8 * 8 * n + faces * (3 * 8 + 8 + 8) + 8 * n, "flops": faces * 90 + n * 30}
    order2 = case["order"] == 1
    mixed = case["eqn"] == "MIXED"
    visc = order2 * (0.5 if mixed else 1.0 if case["eqn"] == "NS" else 0.0)
    per_face = 90 + order2 * (16 + 48) + visc * 130
    per_cell = 40 + order2 * (30 + (40 if case["limiter"] == "SQUEEZE" else 0))
    geo = (7 if order2 else 3) * s + 8
    stages = 3 * case["iterations"]
    moved = 2 * 32 * n * (case["iterations"] if case["kind"] == "coupled" else 1)
    return {"bytes": stages * (8 * s * n + geo * faces + (4 if order2 else 1) * s * n) + moved,
            "flops": stages * (per_face * faces + per_cell * n)}


# ------------------------------------------------------------------------------------------ exact
class _Exact:
    """The method in 64 bits: LSQ gradient, squeeze limiter on the previous stage's face values,
    Rusanov and viscous fluxes, SSP-RK3, as plain torch operations over all faces at once."""

    def __init__(self, grid, opt):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a, k=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(dev, k)  # noqa: E731
        self.o = opt
        self.nc, self.nf = nc, nf = grid.num_cells, grid.num_faces
        p1, p2 = t(grid.fp1, torch.int64) - 1, t(grid.fp2, torch.int64) - 1
        px, py = t(grid.x), t(grid.y)
        self.c1 = c1 = t(grid.fc1, torch.int64) - 1
        raw = t(grid.fc2, torch.int64)
        self.code = torch.where(raw > 0, 0, torch.where(raw == 0, BC[opt["BC1"]], BC[opt["BC2"]]))
        self.inn = raw > 0
        self.i = torch.nonzero(self.inn).reshape(-1)
        self.b = torch.nonzero(~self.inn).reshape(-1)
        self.c2 = torch.where(self.inn, raw - 1, c1)   # boundary faces: a valid index, never used
        xa, ya, xb, yb = px[p1], py[p1], px[p2], py[p2]
        dx, dy = xb - xa, yb - ya
        self.A = torch.hypot(dx, dy)
        self.nx, self.ny = dy / self.A, -dx / self.A
        fx, fy = 0.5 * (xa + xb), 0.5 * (ya + yb)

        def add(v, w=None):   # sum over a cell's faces (w: the value seen from c2, default the same)
            s = torch.zeros(nc, dtype=torch.float64, device=dev).index_add_(0, c1, v)
            return s.index_add_(0, self.c2[self.i], (v if w is None else w)[self.i])

        cnt = add(torch.ones_like(dx))
        mx, my = add(fx) / cnt, add(fy) / cnt          # the vertex mean
        vol, cx, cy = (torch.zeros(nc, dtype=torch.float64, device=dev) for _ in range(3))
        for cell, sel in ((c1, slice(None)), (self.c2[self.i], self.i)):
            gx, gy = mx[cell], my[cell]
            x1, y1, x2, y2 = xa[sel], ya[sel], xb[sel], yb[sel]
            tri = 0.5 * torch.abs(x1 * (y2 - gy) + x2 * (gy - y1) + gx * (y1 - y2))
            vol.index_add_(0, cell, tri)
            cx.index_add_(0, cell, (x1 + x2 + gx) / 3 * tri)
            cy.index_add_(0, cell, (y1 + y2 + gy) / 3 * tri)
        cx, cy = cx / vol, cy / vol
        self.vol = vol
        sgn = 2 * ((fx - cx[c1]) * self.nx + (fy - cy[c1]) * self.ny)
        ox = torch.where(self.inn, cx[self.c2], cx[c1] + sgn * self.nx)   # the other centre (ghost: mirrored)
        oy = torch.where(self.inn, cy[self.c2], cy[c1] + sgn * self.ny)
        self.d1 = (fx - cx[c1], fy - cy[c1])
        self.d2 = (fx - ox, fy - oy)
        self.lx, self.ly = ox - cx[c1], oy - cy[c1]
        sxx, syy, sxy = add(self.lx * self.lx), add(self.ly * self.ly), add(self.lx * self.ly)
        det = sxx * syy - sxy * sxy
        self.I = (sxx / det, syy / det, sxy / det)
        self.dist = torch.hypot(self.lx, self.ly)
        g = opt["gamma"]
        E = opt["P"] / (g - 1) + 0.5 * opt["rho"] * (opt["u"] ** 2 + opt["v"] ** 2)
        self.qinf = torch.tensor([opt["rho"], opt["rho"] * opt["u"], opt["rho"] * opt["v"], E], dtype=torch.float64,
                                 device=dev)[:, None]
        self.dev = dev

    def cellsum(self, v1, v2):
        s = torch.zeros(v1.shape[0], self.nc, dtype=torch.float64, device=self.dev)
        s.index_add_(1, self.c1, v1)
        return s.index_add_(1, self.c2[self.i], v2[:, self.i])

    def prim(self, q):
        u, v = q[1] / q[0], q[2] / q[0]
        return u, v, (self.o["gamma"] - 1) * (q[3] - 0.5 * q[0] * (u * u + v * v))

    def cons(self, rho, u, v, P):
        return torch.stack([rho, rho * u, rho * v, P / (self.o["gamma"] - 1) + 0.5 * rho * (u * u + v * v)])

    def ghosts(self, L, face):
        """Boundary states of faces `face` from the states L on their inner side."""
        code = self.code[face]
        nx, ny = self.nx[face], self.ny[face]
        u, v, P = self.prim(L)
        vn = u * nx + v * ny
        slip = self.cons(L[0], u - 2 * vn * nx, v - 2 * vn * ny, P)
        out = torch.where(code == -1, self.qinf, L)
        out = torch.where(code == -2, slip, out)
        return torch.where(code == -4, self.cons(L[0], -u, -v, P), out)

    def gradient(self, q, faces, initial):
        """Limited gradients; `faces` the previous stage's face states (None: the first stage's -101)."""
        c1, c2, b = self.c1, self.c2, self.b
        d = q[:, c2] - q[:, c1]
        code, inner = self.code[b], q[:, c1[b]]
        src = torch.where(code == -4, q[:, b % self.nc], inner)   # no-slip: the cell numbered like the face
        u, v, P = self.prim(src)
        rho = src[0]
        if initial:
            o = self.o
            rho, u, v, P = (torch.full_like(rho, o[k]) for k in ("rho", "u", "v", "P"))
        nx, ny = self.nx[b], self.ny[b]
        vn = u * nx + v * ny
        gq = torch.where(code == -1, self.qinf, inner)
        gq = torch.where(code == -2, self.cons(rho, u - 2 * vn * nx, v - 2 * vn * ny, P), gq)
        gq = torch.where(code == -4, self.cons(rho, -u, -v, P), gq)
        d[:, b] = gq - inner
        sx, sy = self.cellsum(d * self.lx, d * self.lx), self.cellsum(d * self.ly, d * self.ly)
        Ixx, Iyy, Ixy = self.I
        gx, gy = sx * Iyy - sy * Ixy, sy * Ixx - sx * Ixy
        if self.o["limiter"] == "SQUEEZE":
            lo, hi, phi = q.clone(), q.clone(), torch.ones_like(q)
            e1, e2 = c1[self.i], c2[self.i]
            for a, k in ((e1, e2), (e2, e1)):
                idx = a.expand(4, -1)
                lo.scatter_reduce_(1, idx, q[:, k], "amin")
                hi.scatter_reduce_(1, idx, q[:, k], "amax")
            for cell, sel, side in ((c1, slice(None), 0), (e2, self.i, 1)):
                qf = torch.full_like(q[:, cell], -101.0) if faces is None else faces[side][:, sel]
                qc, mn, mx = q[:, cell], lo[:, cell], hi[:, cell]
                r = torch.where(qf < mn, (mn - qc) / (qf - qc), torch.where(qf > mx, (mx - qc) / (qf - qc), 1.0))
                phi.scatter_reduce_(1, cell.expand(4, -1), r, "amin")
            gx, gy = gx * phi, gy * phi
        return gx, gy

    def stage(self, q, faces, initial):
        """(residual, face states, spectral terms) of state q."""
        o, c1, c2, b = self.o, self.c1, self.c2, self.b
        g = o["gamma"]
        order2 = o["solution_poly_order"] == 1
        nx, ny, A = self.nx, self.ny, self.A
        L, R = q[:, c1], q[:, c2]
        if order2:
            gx, gy = self.gradient(q, faces, initial)
            L = L + gx[:, c1] * self.d1[0] + gy[:, c1] * self.d1[1]
            R = R + gx[:, c2] * self.d2[0] + gy[:, c2] * self.d2[1]
        R[:, b] = self.ghosts(L[:, b], b)
        lu, lv, lP = self.prim(L)
        ru, rv, rP = self.prim(R)
        vl, vr = lu * nx + lv * ny, ru * nx + rv * ny
        F = 0.5 * (torch.stack([L[0] * vl, L[1] * vl + lP * nx, L[2] * vl + lP * ny, vl * (L[3] + lP)])
                   + torch.stack([R[0] * vr, R[1] * vr + rP * nx, R[2] * vr + rP * ny, vr * (R[3] + rP)]))
        spec = torch.abs(0.5 * (vl + vr)) + 0.5 * (torch.sqrt(g * lP / L[0]) + torch.sqrt(g * rP / R[0]))
        F = F - 0.5 * spec * (R - L)
        if order2 and o["eqn"] == "NS":
            a = 0.5 * (L + R)
            au, av, aP = self.prim(a)
            lx, ly = self.lx / self.dist, self.ly / self.dist
            dm = 0.5 * ((gx[:, c1] + gx[:, c2]) * -ny + (gy[:, c1] + gy[:, c2]) * nx)
            dl = (q[:, c2] - q[:, c1]) / self.dist
            gm1 = g - 1
            dQ = [(dl + dm) * lx, (dl + dm) * ly]
            ux = dQ[0][1] - dQ[0][0] * au / a[0]
            vx = dQ[0][2] - dQ[0][0] * av / a[0]
            uy = dQ[1][1] - dQ[1][0] * au / a[0]
            vy = dQ[1][2] - dQ[1][0] * au / a[0]   # the method's own formula has u here
            Px = gm1 * (dQ[0][3] - 0.5 * dQ[0][0] * (au * au + av * av) - a[0] * (au * ux + av * vx))
            Py = gm1 * (dQ[1][3] - 0.5 * dQ[1][0] * (au * au + av * av) - a[0] * (au * uy + av * vy))
            rx, ry = dQ[0][0], dQ[1][0]
            wall = self.code == -4
            cu, cv = q[1][c1] / q[0][c1], q[2][c1] / q[0][c1]
            if initial:
                cu, cv = torch.full_like(cu, o["u"]), torch.full_like(cv, o["v"])
            dn = torch.hypot(*self.d1)
            z = torch.zeros_like(ux)
            for_wall = lambda v, w: torch.where(self.inn, v, torch.where(wall, w, z))  # noqa: E731
            ux, uy = for_wall(ux, -cu / dn * nx), for_wall(uy, -cu / dn * ny)
            vx, vy = for_wall(vx, -cv / dn * nx), for_wall(vy, -cv / dn * ny)
            Px, Py, rx, ry = (torch.where(self.inn, v, z) for v in (Px, Py, rx, ry))
            mu = o["mu"]
            k = mu * (o["R"] * g / (g - 1)) / o["Pr"]
            third = (ux + vy) / 3
            txx, tyy, txy = 2 * mu * (ux - third), 2 * mu * (vy - third), mu * (uy + vx)
            Tx, Ty = (Px * a[0] - rx * aP) / (o["R"] * a[0] ** 2), (Py * a[0] - ry * aP) / (o["R"] * a[0] ** 2)
            V = torch.stack([z, txx * nx + txy * ny, txy * nx + tyy * ny,
                             nx * (au * txx + av * txy + k * Tx) + ny * (au * txy + av * tyy + k * Ty)])
            F = F - V * (self.code != -2)   # slip walls carry no viscous flux
        t = -F * A
        return self.cellsum(t, -t) / self.vol, (L, R), spec * A

    def run(self, q, iterations, initial):
        """`iterations` SSP-RK3 iterations; (state, residual norms of the last stage)."""
        o = self.o
        q = torch.from_numpy(q).to(self.dev).reshape(4, -1)
        faces, first = None, initial
        s0 = (math.hypot(o["u"], o["v"]) + math.sqrt(o["gamma"] * o["P"] / o["rho"])) * self.A
        S = self.cellsum(s0[None], s0[None])[0]
        for _ in range(iterations):
            dt = 2 * o["CFL"] * self.vol / (S.max() if o["time_step_type"] == "GLOBAL" else S)
            r, faces, _s = self.stage(q, faces, first)
            q1 = q + dt * r
            r, faces, _s = self.stage(q1, faces, False)
            q2 = 0.75 * q + 0.25 * q1 + 0.25 * dt * r
            r, faces, s = self.stage(q2, faces, False)
            q = q / 3 + 2 / 3 * q2 + 2 / 3 * dt * r
            S = self.cellsum(s[None], s[None])[0]
            first = False
        return q.reshape(-1).cpu(), torch.sqrt((r * r).sum(1)).cpu()


def exact(case, seed):
    if case["kind"] == "batch":
        if case["cells"] * case["iterations"] > 60_000_000:
            return None   # too long
        runs = []
        for key, c in _batch_solves(case, seed):
            opt, grid = _options(c), _grid(*key)
            E = opt["P"] / (opt["gamma"] - 1) + 0.5 * opt["rho"] * (opt["u"] ** 2 + opt["v"] ** 2)
            q = np.repeat([opt["rho"], opt["rho"] * opt["u"], opt["rho"] * opt["v"], E], grid.num_cells)
            runs.append(_Exact(grid, opt).run(q, c["iterations"], True))
        q = torch.cat([r[0] for r in runs])
        return (q, torch.stack([r[1] for r in runs])) if case["precision"] == "fp64" else q
    grid = _grid(case["mesh"], case["cells"], 1)
    opt = _options(case)
    q = _state(case, opt, grid, seed)
    e = _Exact(grid, opt)
    if case["kind"] == "noalloc":
        return e.stage(torch.from_numpy(q).to(e.dev).reshape(4, -1), None, False)[0].reshape(-1)
    if case["cells"] * case["iterations"] > 60_000_000:
        return None
    q, norms = e.run(q, case["iterations"], False)
    return (q, norms) if case["precision"] == "fp64" else q
