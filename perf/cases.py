"""The assembly work that a user of this library has it do, as timed cases.

A case is a dict of plain values. Its "op" is what the program asks for:

  assemble     mesh -> CSR (pattern and FP64 values), the call of every solver
               step whose mesh changed; "wait" reads the info word back as
               fem_assemble does, otherwise the call only queues work
  system       assemble, body-force load vector, Dirichlet conditions
  upper        lists -> upper-triangle CSR, for a symmetric or Cholesky solver
  reassemble   new coordinates and materials in a known pattern (nonlinear and
               time-stepping solvers)
  ke           the element stiffness matrices alone (element-by-element solvers)
  batch        many independent meshes of all kinds in one call

"kind" is the element kind, nx/ny/nz the cells of the box that the mesh fills.
2-D meshes have jittered nodes, T3 and mixed meshes shuffled element order and
a material per element, as the package's generators make them. Hex20 meshes
have jittered nodes; "shuffle" gives their elements in random order with a
material per element, as an unstructured mesh file would.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "a-lls-matrix-parallel-assembly_b200"))
import fem_alls as fem  # noqa: E402
import meshgen as mg  # noqa: E402

DPN = {"q4": 2, "t3": 2, "mixed": 2, "hex20": 3}


def listed():
    return [
        # the accuracy-test mesh of the Q4 configuration: one small assembly, the caller waiting for it
        {"name": "q4_10x100_wait", "op": "assemble", "kind": "q4", "nx": 100, "ny": 10, "wait": True},
        # the Q4 configuration as a whole linear system: matrix, load vector, boundary conditions
        {"name": "q4_100x100_system", "op": "system", "kind": "q4", "nx": 100, "ny": 100},
        # the T3 configuration: an unstructured plane mesh, 2 M triangles in shuffled order
        {"name": "t3_1000x1000", "op": "assemble", "kind": "t3", "nx": 1000, "ny": 1000},
        # the mixed configuration: Q4 and T3 in one mesh, the largest plane mesh
        {"name": "mixed_1500x1500", "op": "assemble", "kind": "mixed", "nx": 1500, "ny": 1500},
        # a time step of a plane model: values only, pattern kept, ragged box
        {"name": "t3_1001x699_reassemble", "op": "reassemble", "kind": "t3", "nx": 1001, "ny": 699},
        # a small solid part
        {"name": "hex20_9x9x9", "op": "assemble", "kind": "hex20", "nx": 9, "ny": 9, "nz": 9},
        # a solid part of a mesh file: ragged box, shuffled elements, graded material, symmetric storage
        {"name": "hex20_37x21x29_upper", "op": "upper", "kind": "hex20", "nx": 37, "ny": 21, "nz": 29, "shuffle": True},
        # the Hex20 configuration: 262,144 elements, 557 M nonzeros
        {"name": "hex20_64x64x64", "op": "assemble", "kind": "hex20", "nx": 64, "ny": 64, "nz": 64},
        # the tensor-core precision form of the element stiffness
        {"name": "hex20_48x48x48_tc", "op": "assemble", "kind": "hex20", "nx": 48, "ny": 48, "nz": 48, "prec": "tc"},
        # a time step of a solid model
        {"name": "hex20_40x40x40_reassemble", "op": "reassemble", "kind": "hex20", "nx": 40, "ny": 40, "nz": 40},
        # element matrices of a solid model
        {"name": "hex20_39x41x40_ke", "op": "ke", "kind": "hex20", "nx": 39, "ny": 41, "nz": 40},
        # the batched configuration's mix of kinds and sizes, sixteen meshes
        {"name": "batch_16", "op": "batch", "meshes": 16, "emin": 1000, "emax": 50000},
    ]


def draw(rng):
    """A case of the listed ranges: 100 to 3.4 M plane elements, 8 to 262,144 solid ones."""
    def log(lo, hi):
        return lo * (hi / lo) ** rng.random()

    def box2(cells):
        r = log(0.2, 5.0)
        return max(1, round((cells * r) ** 0.5)), max(1, round((cells / r) ** 0.5))

    def box3(cells):
        r, q = log(0.5, 2.0), log(0.5, 2.0)
        side = cells ** (1.0 / 3.0)
        return [max(1, round(side * f)) for f in (r, q, 1.0 / (r * q))]

    op = rng.choice(["assemble", "assemble", "assemble", "system", "upper", "reassemble", "ke", "batch"])
    if op == "batch":
        lo = round(log(200, 4000))
        return {"op": op, "meshes": rng.randint(3, 20), "emin": lo, "emax": round(lo * log(2, 12))}
    kind = rng.choice(["q4", "t3", "mixed", "hex20", "hex20"])
    case = {"op": op, "kind": kind}
    if kind == "hex20":
        nx, ny, nz = box3(log(8, 200_000 if op == "assemble" else 60_000))
        case.update(nx=nx, ny=ny, nz=nz, shuffle=rng.random() < 0.5)
        if op != "system" and rng.random() < 0.25:
            case["prec"] = "tc"
    else:
        nx, ny = box2(log(100, 2_000_000 if op == "assemble" else 700_000))
        case.update(nx=nx, ny=ny)
        if op != "system" and rng.random() < 0.25:
            case["prec"] = "fp32"
    if op == "assemble" and rng.random() < 0.5:
        case["wait"] = True
    return case


# ---- meshes ------------------------------------------------------------------

def hex20_mesh(nx, ny, nz, seed, shuffle):
    """meshgen.hex20_grid's mesh (compact lattice numbering, jittered inside
    nodes) without its Jacobian check: a jitter of 5 % of an edge inverts no
    element. shuffle: random element order and a material per element."""
    r = np.random.default_rng(seed)
    lx, ly, lz = 2 * nx + 1, 2 * ny + 1, 2 * nz + 1
    k, j, i = np.meshgrid(np.arange(lz, dtype=np.int32), np.arange(ly, dtype=np.int32),
                          np.arange(lx, dtype=np.int32), indexing="ij")
    used = ((i & 1) + (j & 1) + (k & 1)) <= 1
    node = (np.cumsum(used.ravel(), dtype=np.int32) - 1)
    i, j, k = i[used], j[used], k[used]
    inside = (i > 0) & (i < lx - 1) & (j > 0) & (j < ly - 1) & (k > 0) & (k < lz - 1)
    h = min(1.0 / nx, 1.0 / ny, 1.0 / nz)
    x, y, z = (c * (0.5 / n) + r.uniform(-0.05 * h, 0.05 * h, c.shape[0]) * inside
               for c, n in ((i, nx), (j, ny), (k, nz)))
    ez, ey, ex = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    base = (2 * ez * ly + 2 * ey) * lx + 2 * ex
    off = mg.HEX20_OFFSETS
    conn = node[base.ravel()[:, None] + ((off[:, 2] * ly + off[:, 1]) * lx + off[:, 0])[None, :]]
    E = nu = None
    if shuffle:
        conn = conn[r.permutation(conn.shape[0])]
        E = r.lognormal(0.0, 0.5, conn.shape[0])
        nu = r.uniform(0.2, 0.4, conn.shape[0])
    return mg.Mesh(mg.HEX20, x, y, z, np.ascontiguousarray(conn), None, E, nu, E0=1.0, nu0=0.3)


def mixed_mesh(nx, ny, seed):
    """meshgen.mixed_grid's mesh with exactly half of the cells Q4, so that every
    seed gives the same number of elements and nonzeros."""
    r = np.random.default_rng(seed)
    x, y = np.meshgrid(np.arange(nx + 1) / nx, np.arange(ny + 1) / ny)
    inside = np.zeros(x.shape, bool)
    inside[1:-1, 1:-1] = True
    h = 0.15 * min(1.0 / nx, 1.0 / ny)
    x, y = ((c + r.uniform(-h, h, c.shape) * inside).ravel() for c in (x, y))
    j, i = np.meshgrid(np.arange(ny, dtype=np.int32), np.arange(nx, dtype=np.int32), indexing="ij")
    n0 = (j * (nx + 1) + i).ravel()
    cell = np.stack([n0, n0 + 1, n0 + nx + 2, n0 + nx + 1], 1)[r.permutation(nx * ny)]
    q, c = cell[:nx * ny // 2], cell[nx * ny // 2:]
    none = np.full((c.shape[0], 1), -1, np.int32)
    conn = np.concatenate([q, np.hstack([c[:, [0, 1, 2]], none]), np.hstack([c[:, [0, 2, 3]], none])])
    types = np.repeat(np.array([mg.Q4, mg.T3], np.uint8), [q.shape[0], 2 * c.shape[0]])
    p = r.permutation(conn.shape[0])
    E, nu = r.lognormal(0.0, 0.5, p.shape[0]), r.uniform(0.2, 0.4, p.shape[0])
    return mg.Mesh(mg.MIXED_2D, x, y, None, np.ascontiguousarray(conn[p]), types[p], E, nu, E0=1.0, nu0=0.3)


def mesh_of(case, seed):
    if case["kind"] == "hex20":
        return hex20_mesh(case["nx"], case["ny"], case["nz"], seed, bool(case.get("shuffle")))
    make = {"q4": mg.q4_grid, "t3": mg.t3_grid, "mixed": mixed_mesh}[case["kind"]]
    return make(case["nx"], case["ny"], seed=seed)


def batch_of(case, seed):
    """Meshes of all kinds in turn, element counts spread over [emin, emax] by their logarithm."""
    n, lo, hi = case["meshes"], case["emin"], case["emax"]
    out = []
    for i in range(n):
        e = lo * (hi / lo) ** (((7 * i) % n) / max(1, n - 1))
        s = seed + 1000 * (i + 1)
        if i % 4 == 3:
            m = max(1, round(e ** (1.0 / 3.0)))
            out.append(hex20_mesh(m, m, m, s, False))
        else:
            m = max(1, round((e / (1.0, 2.0, 1.5)[i % 4]) ** 0.5))
            out.append((mg.q4_grid, mg.t3_grid, mixed_mesh)[i % 4](m, m, seed=s))
    return out


def options(case):
    return fem.opts(precision={"tc": fem.FEM_PREC_TC_F16X3, "fp32": fem.FEM_PREC_FP32}.get(case.get("prec"), 0))


def supports(mesh):
    """Clamped edge or face x = 0 with prescribed displacements on it: (fixed, u)."""
    on = np.repeat(mesh.x == 0.0, mesh.dpn)
    u = np.where(on, 1e-3 * np.cos(np.arange(mesh.num_dofs)), 0.0)
    return on.astype(np.uint8), u


# ---- one pass ------------------------------------------------------------------

def prepare(case, seed):
    """The mesh on the GPU, the handle that a program keeps, and outputs of the pattern's size."""
    st = {"case": case}
    if case["op"] == "batch":
        st["batch"] = fem.Batch(batch_of(case, seed))
        st["batch"].sizes()
        return st
    mesh = mesh_of(case, seed)
    st["mesh"] = mesh
    if case["op"] == "ke":
        st["dev"] = fem.device_arrays(mesh)
        st["opts"] = options(case)
        n = 1890 if mesh.kind == mg.HEX20 else (24 if mesh.kind == mg.T3 else 40)
        st["out"] = torch.empty((mesh.num_elems, n), dtype=torch.float64, device="cuda")
        return st
    a = fem.Assembler(mesh, options(case))
    a.assemble()
    st["asm"] = a
    if case["op"] == "system":
        fixed, u = supports(mesh)
        st["fixed"], st["u"] = torch.from_numpy(fixed).cuda(), torch.from_numpy(u).cuda()
        st["load"] = [0.0] * (mesh.dpn - 1) + [-9.81]
    elif case["op"] == "upper":
        st["capacity"] = int((a.capacity + mesh.num_dofs) // 2)
    elif case["op"] == "reassemble":
        st["re"] = fem.Reassembler(a)
        st["re"].build(a.capacity)
        st["opts"] = options(case)
        st["values"] = torch.empty(a.capacity, dtype=torch.float64, device="cuda")
        # the step's new geometry, in the mesh's device arrays
        r = np.random.default_rng(seed + 77)
        h = 0.01 / max(case["nx"], case["ny"], case.get("nz", 1))
        for k in ("x", "y", "z"):
            if k in a.dev:
                a.dev[k] += torch.from_numpy(r.uniform(-h, h, mesh.num_nodes)).cuda()
    return st


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "batch":
        b = st["batch"]
        b.run()
        return [b.row_ptr, b.col_idx, b.values]
    if op == "ke":
        return fem.element_stiffness(st["mesh"], st["opts"], dev_arrays=st["dev"], out=st["out"])[0]
    a = st["asm"]
    if op == "reassemble":
        st["re"].reassemble(st["values"], st["opts"])
        return st["values"]
    if op == "upper":
        a.scatter()
        return list(a.consolidate_upper(st["capacity"]))
    if case.get("wait"):
        rp, ci, v, _ = a.assemble()
        return [rp, ci, v]
    a.assemble_async()
    if op == "system":
        f, _ = fem.body_force(st["mesh"], st["load"], dev_arrays=a.dev)
        fem.apply_dirichlet(a.row_ptr, a.col_idx, a.values, f, st["fixed"], st["u"])
        return [a.row_ptr, a.col_idx, a.values, f]
    return [a.row_ptr, a.col_idx, a.values]


# ---- what a pass cannot do without ----------------------------------------------

def _size(kind, nx, ny, nz, shuffle):
    """(nodes, elements, ordered node pairs that share an element, input bytes, Ke flops) of a box mesh."""
    if kind == "hex20":
        c = nx * ny * nz
        nodes = (nx + 1) * (ny + 1) * (nz + 1) + sum(a * (b + 1) * (d + 1) for a, b, d in
                                                     ((nx, ny, nz), (ny, nz, nx), (nz, nx, ny)))
        faces = (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1)
        edges = (nx - 1) * (ny - 1) * nz + (nx - 1) * ny * (nz - 1) + nx * (ny - 1) * (nz - 1)
        pairs = 400 * c - 64 * faces + 9 * edges - (nx - 1) * (ny - 1) * (nz - 1)
        # gradients of 20 nodes at 27 points (15 each, J 18) and the 210 upper 3x3 blocks (54 each a point)
        return nodes, c, pairs, 24 * nodes + 80 * c + (16 * c if shuffle else 0), c * 27 * (20 * 33 + 210 * 18)
    c, nodes = nx * ny, (nx + 1) * (ny + 1)
    sides = nx * (ny + 1) + ny * (nx + 1)
    if kind == "q4":
        return nodes, c, nodes + 2 * (sides + 2 * c), 16 * nodes + 16 * c, c * 4 * (40 + 10 * 16)
    if kind == "t3":
        return nodes, 2 * c, nodes + 2 * (sides + c), 16 * nodes + 2 * c * 20, 2 * c * (20 + 6 * 16)
    q = c // 2
    e = q + 2 * (c - q)
    return nodes, e, nodes + 2 * (sides + c + q), 16 * nodes + e * 33, q * 800 + 2 * (c - q) * 116


def work(case):
    op = case["op"]
    if op == "batch":
        b = f = 0.0
        n, lo, hi = case["meshes"], case["emin"], case["emax"]
        for i in range(n):
            e = lo * (hi / lo) ** (((7 * i) % n) / max(1, n - 1))
            m = max(1, round(e ** (1 / 3))) if i % 4 == 3 else max(1, round((e / (1.0, 2.0, 1.5)[i % 4]) ** 0.5))
            w = work({"op": "assemble", "kind": ("q4", "t3", "mixed", "hex20")[i % 4], "nx": m, "ny": m, "nz": m})
            b, f = b + w["bytes"], f + w["flops"]
        return {"bytes": b, "flops": f}
    kind, d = case["kind"], DPN[case["kind"]]
    nodes, elems, pairs, inputs, flops = _size(kind, case["nx"], case["ny"], case.get("nz", 1), bool(case.get("shuffle")))
    nnz = pairs * d * d
    if op == "ke":
        out = elems * 8 * {"hex20": 1890, "t3": 24}.get(kind, 40)
    elif op == "reassemble":
        out = 8 * nnz + 4 * d * nodes
    else:
        if op == "upper":
            nnz = (nnz + d * nodes) // 2
        out = 12 * nnz + 4 * (d * nodes + 1)
        if op == "system":
            out += 8 * d * nodes * 2 + d * nodes  # load vector out, supports in
    return {"bytes": float(inputs + out), "flops": float(flops)}


# ---- the same in plain torch, 64 bits ---------------------------------------------

def _ke_2d(x, y, E, nu, t, conn):
    """[e, npe, npe, 2, 2] plane-stress element stiffness."""
    npe = conn.shape[1]
    xe, ye = x[conn], y[conn]
    if npe == 3:
        pts = [(None, None, 0.5)]
    else:
        g = 0.577350269189626
        pts = [(a, b, 1.0) for a in (-g, g) for b in (-g, g)]
    f = E / (1 - nu * nu)
    d11, d12, d33 = f, f * nu, f * (1 - nu) / 2
    K = torch.zeros((conn.shape[0], npe, npe, 2, 2), dtype=torch.float64, device=x.device)
    for a, b, w in pts:
        if npe == 3:
            dx = torch.tensor([-1.0, 1.0, 0.0], dtype=torch.float64, device=x.device)
            dy = torch.tensor([-1.0, 0.0, 1.0], dtype=torch.float64, device=x.device)
        else:
            dx = 0.25 * torch.tensor([-(1 - b), 1 - b, 1 + b, -(1 + b)], dtype=torch.float64, device=x.device)
            dy = 0.25 * torch.tensor([-(1 - a), -(1 + a), 1 + a, 1 - a], dtype=torch.float64, device=x.device)
        j0, j1, j2, j3 = xe @ dx, ye @ dx, xe @ dy, ye @ dy
        det = j0 * j3 - j1 * j2
        gx = (j3[:, None] * dx - j1[:, None] * dy) / det[:, None]
        gy = (j0[:, None] * dy - j2[:, None] * dx) / det[:, None]
        s = (w * t * det)[:, None, None]
        xx, yy = s * gx[:, :, None] * gx[:, None, :], s * gy[:, :, None] * gy[:, None, :]
        xy, yx = s * gx[:, :, None] * gy[:, None, :], s * gy[:, :, None] * gx[:, None, :]
        e11, e12, e33 = (v[:, None, None] for v in (d11, d12, d33))
        K[..., 0, 0] += e11 * xx + e33 * yy
        K[..., 0, 1] += e12 * xy + e33 * yx
        K[..., 1, 0] += e12 * yx + e33 * xy
        K[..., 1, 1] += e11 * yy + e33 * xx
    return K


def _ke_hex20(X, E, nu, conn):
    """[e, 20, 20, 3, 3] isotropic Hex20 element stiffness."""
    g, wt = (-0.774596669241483, 0.0, 0.774596669241483), (5.0 / 9.0, 8.0 / 9.0, 5.0 / 9.0)
    dn = torch.tensor(np.stack([mg.hex20_shape_derivs(a, b, c) for a in g for b in g for c in g]), device=X.device)
    w = torch.tensor([a * b * c for a in wt for b in wt for c in wt], dtype=torch.float64, device=X.device)
    J = torch.einsum("gin,enj->egij", dn, X[conn])
    det = torch.linalg.det(J)
    G = torch.linalg.solve(J, dn[None].expand(conn.shape[0], -1, -1, -1))       # [e, g, a, n]
    e = conn.shape[0]
    P = G.permute(0, 3, 2, 1).reshape(e, 60, 27)
    M = ((P * (w * det)[:, None, :]) @ P.transpose(1, 2)).reshape(e, 20, 3, 20, 3).permute(0, 1, 3, 2, 4)
    lam, mu = (E * nu / ((1 + nu) * (1 - 2 * nu))), E / (2 * (1 + nu))
    lam, mu = lam[:, None, None, None, None], mu[:, None, None, None, None]
    tr = M.diagonal(dim1=3, dim2=4).sum(-1)[..., None, None] * torch.eye(3, dtype=torch.float64, device=X.device)
    return lam * M + mu * (M.transpose(3, 4) + tr)


def _parts(mesh, dev):
    """(conn, Ke) in chunks: conn [e, npe], Ke [e, npe, npe, dpn, dpn], elements of one type."""
    conn = dev["conn"].long()
    E = dev["E"] if "E" in dev else torch.full((mesh.num_elems,), mesh.E0, dtype=torch.float64, device="cuda")
    nu = dev["nu"] if "nu" in dev else torch.full((mesh.num_elems,), mesh.nu0, dtype=torch.float64, device="cuda")
    if mesh.kind == mg.HEX20:
        X = torch.stack([dev["x"], dev["y"], dev["z"]], 1)
        for s in range(0, mesh.num_elems, 1 << 14):
            c = slice(s, s + (1 << 14))
            yield c, conn[c], _ke_hex20(X, E[c], nu[c], conn[c])
        return
    kinds = [(None, conn.shape[1])] if mesh.types is None else [(dev["types"] == mg.Q4, 4), (dev["types"] == mg.T3, 3)]
    for sel, npe in kinds:
        at = torch.arange(mesh.num_elems, device="cuda") if sel is None else sel.nonzero()[:, 0]
        cn = conn[at][:, :npe]
        yield at, cn, _ke_2d(dev["x"], dev["y"], E[at], nu[at], mesh.thickness, cn)


def _csr(mesh, dev):
    N, d = mesh.num_nodes, mesh.dpn
    conn = dev["conn"].long()
    keys = []
    if mesh.types is None:
        groups = [conn]
    else:
        groups = [conn[dev["types"] == mg.Q4], conn[dev["types"] == mg.T3][:, :3]]
    for c in groups:
        keys.append(torch.unique((c[:, :, None] * N + c[:, None, :]).reshape(-1)))
    keys = torch.unique(torch.cat(keys)) if len(keys) > 1 else keys[0]
    row, col = keys // N, keys % N
    cnt = torch.bincount(row, minlength=N)
    start = torch.cumsum(cnt, 0) - cnt
    rp = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"),
                    torch.cumsum(cnt.repeat_interleave(d) * d, 0)])
    # entry (i, j) of block k of row node n at d * d * start[n] + i * d * cnt[n] + (k - start[n]) * d + j
    at = d * d * start[row] + (torch.arange(keys.numel(), device="cuda") - start[row]) * d
    ci = torch.empty(keys.numel() * d * d, dtype=torch.int32, device="cuda")
    v = torch.zeros(keys.numel() * d * d, dtype=torch.float64, device="cuda")
    for i in range(d):
        for j in range(d):
            ci[at + i * d * cnt[row] + j] = (col * d + j).int()
    for _, c, K in _parts(mesh, dev):
        k = torch.searchsorted(keys, (c[:, :, None] * N + c[:, None, :]).reshape(-1))
        for i in range(d):
            for j in range(d):
                v.index_add_(0, at[k] + i * d * cnt[row[k]] + j, K[..., i, j].reshape(-1))
    return rp.int(), ci, v


def _load(mesh, dev, b):
    N = mesh.num_nodes
    f = torch.zeros((N, mesh.dpn), dtype=torch.float64, device="cuda")
    conn = dev["conn"].long()
    bt = torch.tensor(b, dtype=torch.float64, device="cuda")

    def add(c, wn):
        for d in range(mesh.dpn):
            f[:, d].index_add_(0, c.reshape(-1), (wn * bt[d]).reshape(-1))

    if mesh.kind == mg.HEX20:
        g, wt = (-0.774596669241483, 0.0, 0.774596669241483), (5.0 / 9.0, 8.0 / 9.0, 5.0 / 9.0)
        pts = [(a, b2, c) for a in g for b2 in g for c in g]
        dn = torch.tensor(np.stack([mg.hex20_shape_derivs(*p) for p in pts]), device="cuda")
        w = torch.tensor([a * b2 * c for a in wt for b2 in wt for c in wt], dtype=torch.float64, device="cuda")
        s = np.sign(np.array(mg.HEX20_OFFSETS, float) - 1.0)
        sh = []
        for p in pts:
            q = 1.0 + s * np.array(p)[None, :]
            corner = 0.125 * q.prod(1) * ((s * np.array(p)).sum(1) - 2.0)
            mid = 0.25 * np.where(s == 0, 1.0 - np.array(p)[None, :] ** 2, q).prod(1)
            sh.append(np.where((s != 0).all(1), corner, mid))
        sh = torch.tensor(np.stack(sh), device="cuda")
        X = torch.stack([dev["x"], dev["y"], dev["z"]], 1)
        for k in range(0, mesh.num_elems, 1 << 15):
            c = conn[k:k + (1 << 15)]
            det = torch.linalg.det(torch.einsum("gin,enj->egij", dn, X[c]))
            add(c, (w * det) @ sh)
        return f.reshape(-1)
    t3 = mesh.kind == mg.T3
    x, y, t = dev["x"], dev["y"], mesh.thickness
    sel_q = torch.full((mesh.num_elems,), not t3, device="cuda") if mesh.types is None else dev["types"] == mg.Q4
    c = conn[~sel_q][:, :3]
    if c.shape[0]:
        det = (x[c[:, 1]] - x[c[:, 0]]) * (y[c[:, 2]] - y[c[:, 0]]) - (y[c[:, 1]] - y[c[:, 0]]) * (x[c[:, 2]] - x[c[:, 0]])
        add(c, (t * det / 6.0)[:, None].expand(-1, 3))
    c = conn[sel_q]
    if c.shape[0]:
        g = 0.577350269189626
        sx = torch.tensor([-1.0, 1.0, 1.0, -1.0], dtype=torch.float64, device="cuda")
        sy = torch.tensor([-1.0, -1.0, 1.0, 1.0], dtype=torch.float64, device="cuda")
        wn = 0.0
        for a in (-g, g):
            for b2 in (-g, g):
                dx, dy = 0.25 * sx * (1 + sy * b2), 0.25 * sy * (1 + sx * a)
                det = (x[c] @ dx) * (y[c] @ dy) - (y[c] @ dx) * (x[c] @ dy)
                wn = wn + t * det[:, None] * (0.25 * (1 + sx * a) * (1 + sy * b2))
        add(c, wn)
    return f.reshape(-1)


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        out = [_csr(m, fem.device_arrays(m)) for m in batch_of(case, seed)]
        return [[o[k] for o in out] for k in range(3)]
    mesh = mesh_of(case, seed)
    dev = fem.device_arrays(mesh)
    if op == "ke":
        wide = 1890 if mesh.kind == mg.HEX20 else (24 if mesh.kind == mg.T3 else 40)
        out = torch.zeros((mesh.num_elems, wide), dtype=torch.float64, device="cuda")
        for at, c, K in _parts(mesh, dev):
            iu = torch.triu_indices(c.shape[1], c.shape[1], device="cuda")
            up = K[:, iu[0], iu[1]].reshape(c.shape[0], -1)
            if isinstance(at, slice):
                out[at, :up.shape[1]] = up
            else:
                out[at, :up.shape[1]] = up if up.shape[1] == wide else torch.nn.functional.pad(up, (0, wide - up.shape[1]))[:, :up.shape[1]]
        return out
    if op == "reassemble":
        r = np.random.default_rng(seed + 77)
        h = 0.01 / max(case["nx"], case["ny"], case.get("nz", 1))
        for k in ("x", "y", "z"):
            if k in dev:
                dev[k] += torch.from_numpy(r.uniform(-h, h, mesh.num_nodes)).cuda()
    rp, ci, v = _csr(mesh, dev)
    if op == "reassemble":
        return v
    rows = torch.repeat_interleave(torch.arange(mesh.num_dofs, device="cuda", dtype=torch.int32), (rp[1:] - rp[:-1]).long())
    if op == "upper":
        keep = ci >= rows
        cnt = torch.bincount(rows[keep].long(), minlength=mesh.num_dofs)
        urp = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cumsum(cnt, 0)])
        return [urp.int(), ci[keep], v[keep]]
    if op == "system":
        f = _load(mesh, dev, [0.0] * (mesh.dpn - 1) + [-9.81])
        fixed, u = (torch.from_numpy(t).cuda() for t in supports(mesh))
        fx = fixed.bool()
        fr, fc = fx[rows.long()], fx[ci.long()]
        moved = fc & ~fr
        f.index_add_(0, rows[moved].long(), -v[moved] * u[ci[moved].long()])
        f = torch.where(fx, u, f)
        v = torch.where(fr, (rows == ci).double(), torch.where(fc, torch.zeros_like(v), v))
        return [rp, ci, v, f]
    return [rp, ci, v]
