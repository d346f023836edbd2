"""3D cells whose faces are triangles, quads and pentagons: residual and mesh-coordinate adjoint
against the oracle and its autograd through the geometry."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import fv_oracle as fo
from tests.cases import DUCT3_BC, sst_spec

pytestmark = pytest.mark.gpu


def prisms(nx=6, ny=4, nz=3, seed=0):
    """An extruded box of quads in which every other pair of neighbouring cells is a pentagon and a
    triangle instead (the second quad's half joined to the first), interior nodes jittered."""
    from aquaflux_gb300.mesh import MeshData

    def node(i, j):
        return i * (ny + 1) + j

    cells = []
    for j in range(ny):
        for i in range(0, nx, 2):
            a, b, c = node(i, j), node(i + 1, j), node(i + 2, j)
            d, e, f = node(i + 2, j + 1), node(i + 1, j + 1), node(i, j + 1)
            cells += [[a, b, d, e, f], [b, c, d]] if (i // 2 + j) % 2 else [[a, b, e, f], [b, c, d, e]]
    xy = np.array([(i / nx * 2.0, j / ny) for i in range(nx + 1) for j in range(ny + 1)])
    rng = np.random.default_rng(seed)
    n2, nc2 = len(xy), len(cells)
    nodes = np.concatenate([np.c_[xy, np.full(n2, k / nz)] for k in range(nz + 1)])
    inside = np.all((nodes > 1e-9) & (nodes < np.array([2.0, 1.0, 1.0]) - 1e-9), axis=1)
    nodes[inside] += rng.uniform(-0.02, 0.02, (inside.sum(), 3))
    edges: dict = {}
    for c, poly in enumerate(cells):
        for p, q in zip(poly, poly[1:] + poly[:1]):
            edges.setdefault((min(p, q), max(p, q)), []).append(c)
    inner, outer = [], {name: [] for name in DUCT3_BC}
    for (p, q), cs in sorted(edges.items()):
        side = [n for n, on in (("left", xy[[p, q], 0] == 0), ("right", xy[[p, q], 0] == 2),
                                ("bottom", xy[[p, q], 1] == 0), ("top", xy[[p, q], 1] == 1)) if on.all()]
        for k in range(nz):
            face = [k * n2 + p, k * n2 + q, (k + 1) * n2 + q, (k + 1) * n2 + p]
            own = [c + k * nc2 for c in cs]
            (inner if len(cs) == 2 else outer[side[0]]).append((face, *own))
    for c, poly in enumerate(cells):
        for k in range(nz + 1):
            face = [k * n2 + p for p in poly]
            if 0 < k < nz:
                inner.append((face, c + (k - 1) * nc2, c + k * nc2))
            else:
                outer["back" if k == 0 else "front"].append((face, c + min(k, nz - 1) * nc2))
    faces, patches = list(inner), {}
    for name, of in outer.items():
        patches[name] = np.arange(len(faces), len(faces) + len(of), dtype=np.int32)
        faces += of
    return MeshData(
        nodes=nodes, fn_offsets=np.cumsum([0] + [len(f[0]) for f in faces]).astype(np.int32),
        fn_indices=np.concatenate([f[0] for f in faces]).astype(np.int32),
        owner=np.array([f[1] for f in faces], dtype=np.int32),
        neighbour=np.array([f[2] if len(f) > 2 else -1 for f in faces], dtype=np.int32),
        n_cells=nc2 * nz, patches=patches).validate()


@pytest.mark.parametrize("turbulent", [False, True])
def test_polygonal_faces_match_the_oracle(turbulent):
    from aquaflux_gb300 import fv

    m = prisms()
    counts = np.bincount(np.diff(m.fn_offsets))
    assert (counts[3:6] > 0).all()
    nu, bc, sst = 0.02, DUCT3_BC, None
    if turbulent:
        nu = 1e-3
        bc, sst = sst_spec(3, nu, 0.00375, 1.2, ["bottom", "top", "back", "front"])
    case = fo.make_case(m, mu=nu, rho=1.0, flow_bc=bc, sst=sst)
    fc = fv.FlowCase(fv.DeviceMesh(m), mu=nu, rho=1.0, flow_bc=bc, sst=sst)
    rng = np.random.default_rng(3)
    s = rng.uniform(-0.2, 0.2, (6 if turbulent else 4, m.n_cells))
    s[0] += 1.0
    if turbulent:
        s[4], s[5] = rng.uniform(0.002, 0.006, m.n_cells), rng.uniform(0.8, 2.0, m.n_cells)
    s = s.reshape(-1)
    w = rng.standard_normal(s.size)
    nodes = torch.tensor(m.nodes, dtype=torch.float64, requires_grad=True)
    r = fo.Oracle(case).residual(torch.as_tensor(s), nodes=nodes)
    got = fc.residual(s).cpu().numpy()
    assert np.abs(got - r.detach().numpy()).max() <= 1e-12 * float(r.detach().abs().max())
    (ref,) = torch.autograd.grad((r * torch.as_tensor(w)).sum(), nodes)
    ref, out = ref.numpy(), fc.node_vjp(s, w).cpu().numpy()
    assert np.abs(out - ref).max() <= 1e-10 * np.abs(ref).max()
