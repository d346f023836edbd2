"""The work that a user of this framework has it do, as cases with seeded inputs, and what each comes to.

A case names what is done (``do``) and on which flow (``flow``, with its sizes):

* ``vjp``       residual and its state cotangent, ``FlowCase.vjp(return_residual=True)``: one step of a
                gradient-based calibration or of a training loop through the residual
* ``jvp``       residual and one directional derivative, ``FlowCase.jvp(return_residual=True)``
* ``krylov``    ``FlowCase.linearise`` at an iterate, then Krylov products ``jvp_linearised`` at it: what
                a Newton step asks of the operator
* ``jacobian``  the frozen block Jacobian, fp64 blocks (``BlockJacobian.materialize``)
* ``node_vjp``  the cotangent of every mesh node coordinate (shape sensitivities)
* ``refresh``   one preconditioner refresh of a mixed-precision Newton step and its first application:
                fp32 assembly, the hierarchy's products and ILU(0) factors, one V-cycle
* ``apply``     one application of a refreshed fp32 preconditioner, the V-cycle of each Krylov iteration
* ``ilu``       fp64 ILU(0) of new values, a solve and a transposed solve with it (forward and adjoint
                use of the reference's own preconditioner), unknowns in the mesh's order
* ``solve``     a whole linear solve: 30 iterations of FGMRES on the assembled Jacobian, ILU(0) fp64
* ``renumber``  reverse Cuthill-McKee of a randomly relabelled mesh, host arrays in and out

Flows, with the sizes of this repository's own configurations: ``cavity`` (laminar, 64 x 64 and
below), ``channel`` (3D bump channel with k-omega SST, up to 128^3), ``step`` (2D backward-facing
step with SST and corrected Green-Gauss, ~200k cells) and ``batch`` (laminar 2D channels of uneven
size side by side).  A mesh and its device handle belong to the case and are kept for the next state
on the same case, as a solver or a calibration keeps them; states, tangents and right-hand sides
come from the seed.
"""
import functools
import math

import numpy as np
import torch

from aquaflux_gb300 import fv, mesh as fm, reorder, solve, sparse, workloads
from aquaflux_gb300.amg import AmgPreconditioner
from aquaflux_gb300.ilu0 import Ilu0

F64 = torch.float64


def listed():
    return [
        # the 64 x 64 lid-driven cavity: a small mesh, eleven short launches
        {"name": "cavity-vjp", "do": "vjp", "flow": "cavity", "nx": 64, "ny": 64},
        # the batched calibration sweep: 64 channels of 32^2 to 256^2 cells
        {"name": "batch-vjp", "do": "vjp", "flow": "batch", "nx": 64, "ny": 256},
        # the headline workload, residual and VJP on 2.1M cells with SST
        {"name": "channel-vjp", "do": "vjp", "flow": "channel", "nx": 128, "ny": 128, "nz": 128},
        # the backward-facing step of the validation study: swept gradients, 2D, ragged blocks
        {"name": "step-jvp", "do": "jvp", "flow": "step", "nx": 1300, "ny": 96},
        # a Newton step's Krylov operator (its iterates' linearisation and products)
        {"name": "channel-krylov", "do": "krylov", "flow": "channel", "nx": 96, "ny": 64, "nz": 64},
        # the fp64 preconditioner's operator, on an odd-sized box
        {"name": "channel-jacobian", "do": "jacobian", "flow": "channel", "nx": 80, "ny": 63, "nz": 51},
        # shape gradients of an objective
        {"name": "channel-node-vjp", "do": "node_vjp", "flow": "channel", "nx": 48, "ny": 48, "nz": 48},
        # mixed-precision Newton: what it does once a step, and once a Krylov iteration
        {"name": "channel-refresh", "do": "refresh", "flow": "channel", "nx": 64, "ny": 64, "nz": 64},
        {"name": "channel-apply", "do": "apply", "flow": "channel", "nx": 128, "ny": 96, "nz": 96},
        # the reference's ILU(0) on the cavity's operator: narrow level sets
        {"name": "cavity-ilu", "do": "ilu", "flow": "cavity", "nx": 64, "ny": 64},
        # the cavity's linear solve as a whole
        {"name": "cavity-solve", "do": "solve", "flow": "cavity", "nx": 64, "ny": 64},
        # the channel's renumbering, from host face lists to a host permutation
        {"name": "channel-renumber", "do": "renumber", "flow": "channel", "nx": 128, "ny": 128, "nz": 128},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def box(lo, hi):
        return {"flow": "channel", "nx": size(lo, hi), "ny": size(lo, hi), "nz": size(lo, hi)}

    def plane(flow):
        if flow == "cavity":
            return {"flow": "cavity", "nx": size(16, 96), "ny": size(16, 96)}
        if flow == "step":
            return {"flow": "step", "nx": size(60, 1300), "ny": size(12, 96)}
        return {"flow": "batch", "nx": size(4, 64), "ny": size(48, 256)}

    do = rng.choice(["vjp", "jvp", "krylov", "jacobian", "node_vjp", "refresh", "apply", "ilu", "solve",
                     "renumber"])
    if do in ("vjp", "jvp"):
        where = rng.choice(["cavity", "batch", "channel", "step"])
        return {"do": do, **(box(12, 112) if where == "channel" else plane(where))}
    if do in ("ilu", "solve"):
        return {"do": do, **plane("cavity")}
    if do == "node_vjp":
        return {"do": do, **(box(12, 44) if rng.random() < 0.6 else plane("cavity"))}
    if do == "krylov":
        return {"do": do, **(box(16, 72) if rng.random() < 0.6 else plane("batch"))}
    if do == "jacobian":
        return {"do": do, **(box(16, 64) if rng.random() < 0.6 else plane("cavity"))}
    return {"do": do, **box(20, {"refresh": 64, "apply": 100, "renumber": 112}[do])}


# ---------------------------------------------------------------- what a program keeps
@functools.lru_cache(maxsize=2)
def _flow(flow, nx, ny, nz):
    """The host mesh and case description (``workloads.Workload``)."""
    if flow == "cavity":
        m = fm.structured_grid_2d(nx, ny)
        bc = {"top": ("moving", (1.0, 0.0)), "bottom": ("wall",), "left": ("wall",), "right": ("wall",)}
        return workloads.Workload("cavity", m, 0.01, 1.0, bc, 0, None)
    if flow == "channel":
        return workloads.channel3d(nx, ny, nz)
    if flow == "step":
        return workloads.backward_step(n_step=max(ny // 2, 2), n_channel=ny,
                                       n_upstream=max(nx * 120 // 1300, 4), n_downstream=nx)
    return workloads.batched_channels(nx, n_max=max(ny, 33)).workload


@functools.lru_cache(maxsize=2)
def _handle(flow, nx, ny, nz):
    return _flow(flow, nx, ny, nz).device_case()


def _key(case):
    return case["flow"], case["nx"], case["ny"], case.get("nz", 0)


def _generator(case, seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)


def _state(w, gen):
    """Plug flow (a closed cavity: at rest) with inlet k and omega, 5 % noise on every field."""
    s = torch.as_tensor(w.initial_state(), device="cuda")
    noise = torch.randn(2, s.numel(), dtype=F64, device="cuda", generator=gen)
    return s * (1.0 + 0.05 * noise[0]) + 0.02 * noise[1] * (s == 0)


PRODUCTS = 4  # Krylov products per linearisation here (a Newton step: about twelve)


def prepare(case, seed):
    gen = _generator(case, seed)
    w = _flow(*_key(case))
    if case["do"] == "renumber":
        rng = np.random.default_rng(seed)
        m = fm.permute_cells(fm.structured_grid_3d(case["nx"], case["ny"], case["nz"]),
                             rng.permutation(case["nx"] * case["ny"] * case["nz"]))
        return {"do": "renumber", "owner": m.owner, "neighbour": m.neighbour, "n": m.n_cells}
    c = _handle(*_key(case))
    n = c.n_unknowns

    def vector(k=None):
        return torch.randn(*((n,) if k is None else (k, n)), dtype=F64, device="cuda", generator=gen)

    st = {"do": case["do"], "case": c, "s": _state(w, gen)}
    if case["do"] in ("vjp", "jvp", "node_vjp", "refresh", "apply", "solve"):
        st["v"] = vector()
    if case["do"] == "krylov":
        st["v"] = vector(PRODUCTS)
    if case["do"] == "jacobian":
        st["jac"] = solve.BlockJacobian(c)
    if case["do"] in ("refresh", "apply"):
        st["pc"] = AmgPreconditioner(solve.BlockJacobian(c, precision=32), 32)
    if case["do"] == "apply":
        st["pc"].refresh(st["s"])
    if case["do"] in ("ilu", "solve"):
        st["jac"] = jac = solve.BlockJacobian(c)
        jac.materialize(st["s"])
    if case["do"] == "ilu":
        st["ilu"] = Ilu0.from_csr(jac.indptr, jac.indices, jac.values, block_size=jac.b)
        st["rhs"] = vector()
    if case["do"] == "solve":
        st["pc"] = solve.IluPreconditioner(jac, 64)
        st["pc"].refresh(st["s"])
        st["ws"] = solve.KrylovWorkspace(n, 30)
    return st


def run(st):
    do = st["do"]
    if do == "renumber":
        return reorder.rcm_permutation(st["owner"], st["neighbour"], st["n"])
    c, s = st["case"], st["s"]
    if do == "vjp":
        return c.vjp(s, st["v"], return_residual=True)
    if do == "jvp":
        return c.jvp(s, st["v"], return_residual=True)
    if do == "krylov":
        r = c.linearise(s)
        return [r] + [c.jvp_linearised(s, v) for v in st["v"]]
    if do == "jacobian":
        return st["jac"].materialize(s)
    if do == "node_vjp":
        return c.node_vjp(s, st["v"])
    if do == "refresh":
        st["pc"].refresh(s)
        return st["pc"].apply(st["v"])
    if do == "apply":
        return st["pc"].apply(st["v"])
    if do == "ilu":
        f = st["ilu"]
        f.refactor(st["jac"].values)
        return f.solve(st["rhs"]), f.solve(st["rhs"], transpose=True)
    jac, n, b = st["jac"], st["jac"].n, st["jac"].b

    def matvec(x):  # the state's field-major layout around the cell-major operator
        y = sparse.bsr_spmv(jac.d_indptr, jac.d_indices, jac.values, b, x.view(b, n).t().reshape(-1))
        return y.view(n, b).t().reshape(-1)

    return solve.fgmres(matvec, st["v"], st["pc"].apply, rtol=0.0, restart=30, maxiter=30,
                        workspace=st["ws"]).x


def work(case):
    """Bytes: every input and output once -- the fields, and of the mesh the face-to-cell lists, face area
    vectors and centroids, cell volumes and centroids (nodes where geometry is differentiated).
    Flops: additions and multiplications of the discretisation, each face and cell once."""
    flow, nx, ny, nz = _key(case)
    if flow == "batch":
        m = _flow(flow, nx, ny, nz).mesh
        nc, nf = m.n_cells, m.n_faces
    elif flow == "channel":
        nc, nf = nx * ny * nz, 3 * nx * ny * nz + nx * ny + ny * nz + nx * nz
    else:
        nc = nx * ny if flow == "cavity" else _flow(flow, nx, ny, nz).mesh.n_cells
        nf = 2 * nc + nx + ny
    dim, sst = (3, True) if flow == "channel" else (2, flow == "step")
    b = dim + 1 + 2 * sst
    n = b * nc
    mesh = nf * (8 + 16 * dim) + nc * (8 + 8 * dim + (8 + 8 * dim) * sst)
    nnzb = nc + 2 * nf
    per_face = 40 + 30 * dim + 24 * dim * dim * 0.5 + 50 * sst  # the residual's, cells' part included
    do = case["do"]
    if do == "vjp":
        return {"bytes": mesh + 4 * 8 * n, "flops": 2.5 * per_face * nf}
    if do == "jvp":
        sweeps = 3 * 12 * dim * b if flow == "step" else 0
        return {"bytes": mesh + 4 * 8 * n, "flops": 2.0 * (per_face + sweeps) * nf}
    if do == "krylov":
        return {"bytes": mesh + (2 + 2 * PRODUCTS) * 8 * n, "flops": (1 + PRODUCTS) * per_face * nf}
    if do == "jacobian":
        return {"bytes": mesh + 8 * n + 8 * b * b * nnzb, "flops": (per_face + 4 * b * b) * nf}
    if do == "node_vjp":
        return {"bytes": mesh + 2 * 8 * n + 8 * dim * nc, "flops": 5.0 * per_face * nf}
    if do == "refresh":
        return {"bytes": mesh + 3 * 8 * n + 4 * b * b * nnzb, "flops": nnzb * (2 * b ** 3 + 4 * b * b)}
    if do == "apply":  # two smoothing sweeps (the factors) and two products on the finest level
        return {"bytes": 4 * 4 * b * b * nnzb + 2 * 8 * n, "flops": 4 * 2 * b * b * nnzb}
    if do == "ilu":
        return {"bytes": 8 * b * b * nnzb + 3 * 8 * n, "flops": nnzb * (2 * b ** 3 + 8 * b * b)}
    if do == "solve":
        return {"bytes": 2 * 8 * b * b * nnzb + 32 * 8 * n,
                "flops": 30 * (4 * b * b * nnzb + 4 * 16 * n)}
    return {"bytes": 8 * nf + 8 * nc, "flops": 0}


# ---------------------------------------------------------------- the same results in plain torch
A1, BS, KAPPA, EW, B1, B2 = 0.31, 0.09, 0.41, 9.8, 3.0 / 40.0, 0.0828
SK1, SW1, SK2, SW2, AL1, AL2 = 0.85, 0.5, 1.0, 0.856, 5.0 / 9.0, 0.44
YLAM = 11.0
for _ in range(10):
    YLAM = math.log(EW * YLAM) / KAPPA


def _sqrt(x):
    ok = x > 0.0
    return torch.where(ok, torch.sqrt(torch.where(ok, x, 1.0)), 0.0)


def _pos(x):
    return torch.clamp(x, min=0.0)


class _Plain:
    """The discretisation in 64-bit torch operations on whole arrays, differentiated by autograd."""

    def __init__(self, w):
        m = self.m = w.mesh
        self.w, self.dim, self.nc, self.nf = w, m.dim, m.n_cells, m.n_faces

        def dev(a, t=torch.long):
            return torch.as_tensor(np.asarray(a), dtype=t, device="cuda")

        self.o, nb = dev(m.owner), dev(m.neighbour)
        self.inner = nb >= 0
        self.n = torch.where(self.inner, nb, self.o)
        off = np.asarray(m.fn_offsets, dtype=np.int64)
        cnt = np.diff(off)
        face = np.repeat(np.arange(self.nf), cnt)
        at = np.arange(off[-1]) - off[face]
        self.fn, self.fn_face = dev(m.fn_indices), dev(face)
        self.fn_next, self.fn_cnt = dev(off[face] + (at + 1) % cnt[face]), dev(cnt, F64)
        self.nodes = dev(m.nodes, F64)
        t = fv.case_tables(m, w.flow_bc, w.sst)
        self.t = {k: dev(v, F64 if np.asarray(v).dtype == np.float64 else torch.long) for k, v in t.items()}
        self.mu = dev(np.broadcast_to(np.asarray(w.mu, dtype=np.float64), (self.nc,)).copy(), F64)
        if w.sst is not None:
            self.wf = torch.nonzero(self.t["sst_wall"]).reshape(-1)
            self.wc = torch.unique(self.o[self.wf])
            self.near = None

    def add(self, own, nb):
        z = torch.zeros((self.nc,) + own.shape[1:], dtype=F64, device="cuda")
        keep = self.inner.reshape((-1,) + (1,) * (own.dim() - 1))
        return z.index_add(0, self.o, own).index_add(0, self.n, torch.where(keep, nb, 0.0))

    def geometry(self, nodes):
        dim, one = self.dim, torch.ones(self.nf, dtype=F64, device="cuda")
        if dim == 2:
            v = nodes[self.fn].reshape(self.nf, 2, 2)
            d = v[:, 1] - v[:, 0]
            xf, S = 0.5 * (v[:, 0] + v[:, 1]), torch.stack([d[:, 1], -d[:, 0]], 1)
            A = torch.linalg.norm(S, dim=1)
            nrm = S / A[:, None]
        else:
            def per_face(x):
                return torch.zeros((self.nf,) + x.shape[1:], dtype=F64, device="cuda").index_add(
                    0, self.fn_face, x)

            pb = nodes[self.fn]
            pc = pb[self.fn_next]
            pa = (per_face(pb) / self.fn_cnt[:, None])[self.fn_face]
            tri = 0.5 * torch.linalg.cross(pb - pa, pc - pa, dim=-1)
            S = per_face(tri)
            A = torch.linalg.norm(S, dim=1)
            nrm = S / A[:, None]
            xf = per_face((tri * nrm[self.fn_face]).sum(-1)[:, None] * (pa + pb + pc) / 3.0) / A[:, None]
        mid = self.add(xf, xf) / self.add(one, one)[:, None]
        out = ((xf - mid[self.o]) * nrm).sum(-1)
        nrm = nrm * torch.where(out < 0, -1.0, 1.0)[:, None]
        lo, ln = xf - mid[self.o], xf - mid[self.n]
        fo, fn = (lo * nrm).sum(-1) * A, (ln * nrm).sum(-1) * A
        V = self.add(fo, -fn) / dim
        xc = self.add(fo[:, None] * lo, -fn[:, None] * ln) / ((dim + 1) * V)[:, None] + mid
        g = self.g = {"A": A, "nrm": nrm, "xf": xf, "V": V, "xc": xc}
        d = g["d"] = xc[self.n] - xc[self.o]
        inner = self.inner
        g["g"] = torch.where(inner, ((xf - xc[self.o]) * d).sum(-1) /
                             torch.where(inner, (d * d).sum(-1), 1.0), 0.0)
        g["dp"], g["dn"] = xf - xc[self.o], xf - xc[self.n]
        g["dpn"], g["dnn"] = (g["dp"] * nrm).sum(-1), (g["dn"] * nrm).sum(-1)
        g["nd"] = torch.where(inner, (d * nrm).sum(-1), g["dpn"])
        g["skew"] = xf - (xc[self.o] + d * g["g"][:, None])
        g["tp"], g["tn"] = g["dp"] - nrm * g["dpn"][:, None], g["dn"] - nrm * g["dnn"][:, None]

    def face(self, q):
        a = self.g["g"].reshape((-1,) + (1,) * (q.dim() - 1))
        return (1.0 - a) * q[self.o] + a * q[self.n]

    def grad(self, phi, bval):
        g, scheme = self.g, self.w.gradient
        S = g["nrm"] * g["A"][:, None]
        q = S * torch.where(self.inner, self.face(phi), bval)[:, None]
        rhs, V = self.add(q, -q), g["V"][:, None]
        x = rhs / V
        for _ in range((scheme["sweeps"] - 1) if scheme else 0):
            a = g["g"]
            wq = (1.0 - a) * (g["skew"] * x[self.o]).sum(-1) + a * (g["skew"] * x[self.n]).sum(-1)
            c = S * torch.where(self.inner, wq, 0.0)[:, None]
            x = x + (rhs - (x * V - self.add(c, -c))) / V
        return x

    def wall_distance(self):
        xc, xw = self.g["xc"], self.g["xf"][self.wf]
        if self.near is None:
            with torch.no_grad():
                step = max(1, int(2e8 / xw.shape[0]))
                self.near = torch.cat([(((xc[i:i + step, None, 0] - xw[None, :, 0]) ** 2) + sum(
                    (xc[i:i + step, None, j] - xw[None, :, j]) ** 2 for j in range(1, self.dim)))
                    .argmin(1) for i in range(0, self.nc, step)])
        dv = xc - xw[self.near]
        d = torch.sqrt((dv * dv).sum(-1))
        return d, self.grad(d, torch.where(self.t["sst_wall"] > 0, 0.0, d[self.o]))

    @staticmethod
    def y_star(nu, d, k):
        return BS ** 0.25 * _sqrt(_pos(k)) * d / nu

    def weight(self, nu, d, k):
        return torch.tanh((self.y_star(nu, d, k) / YLAM) ** 4)

    def nut_wall(self, nu, d, k):
        y = self.y_star(nu, d, k)
        r = y * KAPPA / torch.log(EW * torch.clamp(y, min=YLAM)) - 1.0
        return nu * torch.where(y > YLAM, r, 0.0)

    def split(self, state):
        f = state.reshape(-1, self.nc)
        return [f[i] for i in range(f.shape[0])]

    def frozen(self, state):
        """Gradients, closure and V / a_P of a state, for :meth:`fluxes`."""
        g, t, w, dim, o, n = self.g, self.t, self.w, self.dim, self.o, self.n
        q = self.split(state)
        u, p = q[:dim], q[dim]
        kind, A, nrm, V = t["flow_kind"], g["A"], g["nrm"], g["V"]
        rho = w.rho
        h = {"bu": [torch.where(kind == 3, u[i][o], torch.where((kind == 1) | (kind == 2),
                                                                t["flow_vel"][:, i], 0.0))
                    for i in range(dim)]}
        h["gu"] = [self.grad(u[i], h["bu"][i]) for i in range(dim)]
        h["gp"] = self.grad(p, torch.where(kind == 3, t["flow_p"], torch.where(kind >= 0, p[o], 0.0)))
        mu = self.mu
        visc = mu
        if w.sst is not None:
            k, om = q[dim + 1], q[dim + 2]
            nu, wc, wf = mu / rho, self.wc, self.wf
            ow = o[wf]
            d, dg = self.wall_distance()
            h["d"] = d

            def bval(phi, name):
                kd = t[name + "_kind"]
                return torch.where(kd == 0, t[name + "_val"], torch.where(kd == 1, phi[o], 0.0))

            gu = torch.stack(h["gu"], 1)
            s = 0.5 * (gu + gu.transpose(1, 2))
            S = _sqrt(2.0 * (s * s).sum((1, 2)))
            wt = self.weight(nu[wc], d[wc], k[wc])
            S = S.index_copy(0, wc, (1 - wt) * S[wc] +
                             wt * BS ** 0.25 * _sqrt(_pos(k[wc])) / (KAPPA * d[wc]))
            h["gk"], h["gw"] = self.grad(k, bval(k, "k")), self.grad(om, bval(om, "omega"))
            vis, kp = 6.0 * nu[wc] / (B1 * d[wc] ** 2), _pos(k[wc])
            c = BS ** 0.25 * KAPPA
            lg = _sqrt(kp) / (c * d[wc])
            ww = torch.sqrt(vis * vis + lg * lg)
            sk = _sqrt(kp)
            dsk = torch.where(sk > 0, 0.5 / torch.where(sk > 0, sk, 1.0), 0.0)
            dd = (vis * (-2.0 * vis / d[wc]) + lg * (-lg / d[wc])) / ww
            imposed = dg[wc] * dd[:, None] + h["gk"][wc] * (lg / ww * dsk / (c * d[wc]))[:, None]
            h["gwi"] = h["gw"].index_copy(0, wc, imposed)
            kp = _pos(k)
            dot = (h["gk"] * h["gwi"]).sum(-1)
            cd = torch.clamp(2.0 * SW2 * dot / om, min=1e-10)
            c1, vt = _sqrt(kp) / (BS * om * d), 500.0 * nu / (d * d * om)
            F1 = torch.tanh(torch.minimum(torch.maximum(c1, vt), 4.0 * SW2 * kp / (cd * d * d)) ** 4)
            F2 = torch.tanh(torch.maximum(2.0 * c1, vt) ** 2)
            nut = A1 * kp / torch.maximum(A1 * om, S * F2)
            h.update(S=S, F1=F1, nut=nut, dot=dot)
            h["gamma"] = [nu + (F1 * SK1 + (1 - F1) * SK2) * nut, nu + (F1 * SW1 + (1 - F1) * SW2) * nut]
            slip = torch.stack([u[i][ow] - h["bu"][i][wf] for i in range(dim)], 1)
            z = torch.zeros(self.nc, dtype=F64, device="cuda")
            h["shear"] = (z.index_add(0, ow, _sqrt((slip * slip).sum(-1)) / d[ow] * A[wf])[wc] /
                          z.index_add(0, ow, A[wf])[wc])
            visc = mu + rho * nut
        h["visc"] = visc
        est = self.estimate(h, [x[o] for x in u], [x[n] for x in u])
        go, gn = visc[o], visc[n]
        vc = go * A / torch.where(self.inner, g["dpn"] - go / gn * g["dnn"], g["dpn"])
        vo = self.boundary_viscosity(h, [x[o] for x in q]) * A / g["nd"]
        own = torch.where(self.inner, vc + _pos(est), torch.where(
            (kind == 0) | (kind == 1), vo, torch.where(kind == 2, vo + _pos(est), torch.where(
                kind == 3, _pos(est), 0.0))))
        h["dco"] = V / self.add(own, vc + _pos(-est))
        return h

    def boundary_viscosity(self, h, qo):
        visc, kind = h["visc"][self.o], self.t["flow_kind"]
        if self.w.sst is None:
            return visc
        ow, wf = self.o[self.wf], self.wf
        wall = torch.zeros(self.nf, dtype=F64, device="cuda").index_copy(
            0, wf, self.nut_wall(self.mu[ow] / self.w.rho, h["d"][ow], qo[self.dim + 1][wf]))
        return torch.where((kind == 0) | (kind == 1), self.mu[self.o] + self.w.rho * wall, visc)

    def estimate(self, h, uo, un):
        g, est = self.g, 0.0
        for i in range(self.dim):
            gf = self.face(h["gu"][i])
            est = est + ((1 - g["g"]) * uo[i] + g["g"] * un[i] + (gf * g["skew"]).sum(-1)) * g["nrm"][:, i]
        return self.w.rho * est * g["A"]

    def fluxes(self, h, qo, qn):
        """Face fluxes of every field from the owner's and the neighbour's values, `h` held."""
        g, t, w, dim, o, n, inner = self.g, self.t, self.w, self.dim, self.o, self.n, self.inner
        A, nrm, kind, rho = g["A"], g["nrm"], t["flow_kind"], w.rho
        uo, un, po, pn = qo[:dim], qn[:dim], qo[dim], qn[dim]
        bu = [torch.where(kind == 3, uo[i], h["bu"][i]) for i in range(dim)]
        damp = ((pn - po) - (self.face(h["gp"]) * g["d"]).sum(-1)) / g["nd"]
        nn = (nrm * nrm).sum(-1)
        inside = self.estimate(h, uo, un) - rho * A * nn * self.face(h["dco"]) * damp
        inlet = rho * A * sum(bu[i] * nrm[:, i] for i in range(dim))
        outlet = rho * A * (sum(uo[i] * nrm[:, i] for i in range(dim)) - nn * h["dco"][o] * (
            (t["flow_p"] - po) / g["nd"] - (h["gp"][o] * nrm).sum(-1)))
        mdot = torch.where(inner, inside, torch.where(kind == 2, inlet, torch.where(kind == 3, outlet, 0.0)))
        pf = torch.where(inner, (1 - g["g"]) * po + g["g"] * pn + (self.face(h["gp"]) * g["skew"]).sum(-1),
                         torch.where(kind == 3, t["flow_p"], torch.where(kind >= 0, po, 0.0)))

        def transport(fo, fn, b, gr, gam, gam_b, flux):
            co, cn = (gr[o] * g["tp"]).sum(-1), (gr[n] * g["tn"]).sum(-1)
            den = torch.where(inner, g["dpn"] - gam[o] / gam[n] * g["dnn"], g["dpn"])
            diff = torch.where(inner, gam[o], gam_b) * torch.where(inner, fn - fo + cn - co, b - fo - co) / den
            return flux * torch.where(flux >= 0, fo, torch.where(inner, fn, b)) - diff * A

        bvisc = self.boundary_viscosity(h, qo)
        out = [transport(uo[i], un[i], bu[i], h["gu"][i], h["visc"], bvisc, mdot) + pf * nrm[:, i] * A
               for i in range(dim)] + [mdot]
        if w.sst is not None:
            nu = self.mu / rho
            for s, name in enumerate(("k", "omega")):
                gr, gam = h["gk" if s == 0 else "gw"], h["gamma"][s]
                fo, fn = qo[dim + 1 + s], qn[dim + 1 + s]
                kd = t[name + "_kind"]
                b = torch.where(kd == 0, t[name + "_val"],
                                torch.where(kd == 1, fo + (gr[o] * g["tp"]).sum(-1), 0.0))
                gb = gam[o]
                if s == 0:
                    ow = o[self.wf]
                    gb = gb.index_copy(0, self.wf, (1 - self.weight(nu[ow], h["d"][ow], fo[self.wf])) *
                                       gb[self.wf])
                out.append(transport(fo, fn, b, gr, gam, gb, mdot / rho))
        return out

    def sources(self, h, k, om, rk, rw):
        wc, nu, V = self.wc, self.mu / self.w.rho, self.g["V"]
        d, kw = h["d"][self.wc], k[self.wc]
        S, F1, nut = h["S"], h["F1"], h["nut"]
        limit = 10.0 * BS * _pos(k) * om
        lim = torch.minimum(nut * S * S, limit)
        wt = self.weight(nu[wc], d, kw)
        pw = (nu[wc] + self.nut_wall(nu[wc], d, kw)) * h["shear"] * BS ** 0.25 * _sqrt(_pos(kw)) / (KAPPA * d)
        lim = lim.index_copy(0, wc, (1 - wt) * lim[wc] + wt * pw)
        vis, lg = 6.0 * nu[wc] / (B1 * d * d), _sqrt(_pos(kw)) / (BS ** 0.25 * KAPPA * d)
        ow = torch.sqrt(vis * vis + lg * lg)
        rk = rk - lim * V + BS * k * om.index_copy(0, wc, ow) * V
        cap = limit / torch.clamp(nut, min=1e-30)
        rw = rw + V * ((F1 * B1 + (1 - F1) * B2) * om * om - (F1 * AL1 + (1 - F1) * AL2) * torch.minimum(
            S * S, cap) - 2.0 * (1 - F1) * SW2 * h["dot"] / om)
        return rk, rw.index_copy(0, wc, om[wc] - ow)

    def residual(self, state):
        h, q, dim = self.frozen(state), self.split(state), self.dim
        r = [self.add(f, -f) for f in self.fluxes(h, [x[self.o] for x in q], [x[self.n] for x in q])]
        if self.w.pressure_pin is not None:
            r[dim] = r[dim].index_copy(0, torch.tensor([self.w.pressure_pin], device="cuda"),
                                       q[dim][self.w.pressure_pin].reshape(1))
        if self.w.sst is not None:
            r[dim + 1], r[dim + 2] = self.sources(h, q[dim + 1], q[dim + 2], r[dim + 1], r[dim + 2])
        return torch.cat(r)

    def jacobian(self, state):
        """Blocks of the frozen Jacobian by (row cell, column cell), columns ascending: (indptr, indices, blocks)."""
        with torch.no_grad():
            h = self.frozen(state)
        q = self.split(state)
        b, o, n, inner, nc = len(q), self.o, self.n, self.inner, self.nc

        def side(own):
            cols = []
            for j in range(b):
                qo, qn = [x[o] for x in q], [x[n] for x in q]
                x = (qo if own else qn)[j].clone().requires_grad_(True)
                (qo if own else qn)[j] = x
                fl = self.fluxes(h, qo, qn)
                cols.append(torch.stack([torch.autograd.grad(f.sum(), x, retain_graph=True)[0]
                                         if f.requires_grad else torch.zeros_like(x) for f in fl], 1))
            return torch.stack(cols, 2)  # (face, flux, unknown)

        D, E = side(True), side(False)
        oi, ni = o[inner], n[inner]
        rows = torch.cat([torch.arange(nc, device="cuda"), oi, ni])
        cols = torch.cat([torch.arange(nc, device="cuda"), ni, oi])
        dia = torch.zeros(nc, b, b, dtype=F64, device="cuda").index_add(0, o, D).index_add(0, ni, -E[inner])
        off_o, off_n = E[inner], -D[inner]
        if self.w.sst is not None:
            k = q[b - 2].clone().requires_grad_(True)
            om = q[b - 1].clone().requires_grad_(True)
            zero = torch.zeros_like(k)
            rk, rw = self.sources(h, k, om, zero, zero)
            wall = torch.zeros(nc, dtype=torch.bool, device="cuda")
            wall[self.wc] = True
            dia[wall, b - 1] = 0.0
            off_o[wall[oi], b - 1] = 0.0
            off_n[wall[ni], b - 1] = 0.0
            for i, r in ((b - 2, rk), (b - 1, rw)):
                for j, x in ((b - 2, k), (b - 1, om)):
                    dia[:, i, j] += torch.autograd.grad(r.sum(), x, retain_graph=True)[0]
        if self.w.pressure_pin is not None:
            c, i = self.w.pressure_pin, self.dim
            dia[c, i] = 0.0
            dia[c, i, i] = 1.0
            off_o[oi == c, i] = 0.0
            off_n[ni == c, i] = 0.0
        order = torch.argsort(rows * nc + cols)
        blocks = torch.cat([dia, off_o, off_n])[order]
        ptr = torch.zeros(nc + 1, dtype=torch.long, device="cuda")
        ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=nc), 0)
        return ptr, cols[order], blocks


class _PlainIlu:
    """Block ILU(0) with numpy, row by row."""

    def __init__(self, ptr, idx, blocks):
        self.ptr, self.idx = ptr.cpu().numpy(), idx.cpu().numpy()
        a = self.a = blocks.cpu().numpy().copy()
        n, self.b = self.ptr.size - 1, a.shape[1]
        self.row = [{int(self.idx[p]): p for p in range(self.ptr[i], self.ptr[i + 1])} for i in range(n)]
        self.inv = np.empty((n, self.b, self.b))
        for i in range(n):
            for j in [j for j in self.row[i] if j < i]:
                lij = a[self.row[i][j]] = a[self.row[i][j]] @ self.inv[j]
                for k, p in self.row[j].items():
                    if k > j and k in self.row[i]:
                        a[self.row[i][k]] -= lij @ a[p]
            self.inv[i] = np.linalg.inv(a[self.row[i][i]])

    def solve(self, r, transpose=False):
        n = self.ptr.size - 1
        y, a, row, inv = r.reshape(n, self.b).copy(), self.a, self.row, self.inv
        if not transpose:
            for i in range(n):
                for j, p in row[i].items():
                    if j < i:
                        y[i] -= a[p] @ y[j]
            for i in reversed(range(n)):
                for j, p in row[i].items():
                    if j > i:
                        y[i] -= a[p] @ y[j]
                y[i] = inv[i] @ y[i]
            return y.reshape(-1)
        for i in range(n):  # (D + U)^T, then (I + L)^T
            y[i] = inv[i].T @ y[i]
            for j, p in row[i].items():
                if j > i:
                    y[j] -= a[p].T @ y[i]
        for i in reversed(range(n)):
            for j, p in row[i].items():
                if j < i:
                    y[j] -= a[p].T @ y[i]
        return y.reshape(-1)


def exact(case, seed):
    do = case["do"]
    if do in ("refresh", "apply", "renumber"):  # a sequential elimination over the whole channel; whole numbers
        return None
    st = prepare(case, seed)
    w = _flow(*_key(case))
    ref, s = _Plain(w), st["s"]
    if do == "node_vjp":
        nodes = ref.nodes.clone().requires_grad_(True)
        ref.geometry(nodes)
        return torch.autograd.grad(ref.residual(s), nodes, st["v"])[0]
    with torch.no_grad():
        ref.geometry(ref.nodes)
    if do in ("ilu", "solve"):
        ptr, idx, blocks = ref.jacobian(s)
        f = _PlainIlu(ptr, idx, blocks)
    if do == "ilu":
        r = st["rhs"].cpu().numpy()
        return f.solve(r), f.solve(r, True)
    if do == "jacobian":
        return ref.jacobian(s)[2].reshape(-1)
    if do == "solve":
        n, b = ref.nc, blocks.shape[1]
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), ptr[1:] - ptr[:-1])

        def product(x):
            y = torch.zeros(n, b, dtype=F64, device="cuda")
            return y.index_add(0, rows, (blocks @ x.view(n, b)[idx][:, :, None])[:, :, 0]).reshape(-1)

        r = st["v"].view(b, n).t().reshape(-1)
        beta = torch.linalg.norm(r)
        V, Z, H = [r / beta], [], torch.zeros(31, 30, dtype=F64, device="cuda")
        for j in range(30):
            Z.append(torch.as_tensor(f.solve(V[j].cpu().numpy()), device="cuda"))
            y, B = product(Z[j]), torch.stack(V)
            for _ in range(2):
                c = B @ y
                y = y - c @ B
                H[:j + 1, j] += c
            H[j + 1, j] = torch.linalg.norm(y)
            V.append(y / H[j + 1, j])
        e = torch.zeros(31, 1, dtype=F64, device="cuda")
        e[0] = beta
        x = torch.linalg.lstsq(H, e).solution[:, 0] @ torch.stack(Z)
        return x.view(n, b).t().reshape(-1)
    x = s.clone().requires_grad_(True)
    r = ref.residual(x)
    if do == "vjp":
        return r.detach(), torch.autograd.grad(r, x, st["v"])[0]
    u = torch.zeros_like(r, requires_grad=True)
    (g,) = torch.autograd.grad(r, x, u, create_graph=True)
    v = st["v"].reshape(-1, x.numel())
    out = [torch.autograd.grad(g, u, t, retain_graph=True)[0] for t in v]
    return (r.detach(), out[0]) if do == "jvp" else [r.detach()] + out
