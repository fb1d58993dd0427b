"""The thread-per-node row lists of the 2-D kinds (rows2d.cu) at the sizes where
they change path, through the C ABI against the oracle: rows at the limits of
the shared-memory sums (8 columns besides the diagonal), of the chunk (14
columns, 14 elements) and of the element list kept in the row's own storage
(126 elements); node counts around a CTA's 64; elements with a repeated node;
output buffers that are not aligned for the wide copy. Pattern bit for bit,
values within 1e-12 of max(|K_ij|, sqrt(|K_ii K_jj|))."""
import ctypes as C

import numpy as np
import pytest

from conftest import diag_scale

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def _compare(oracle_mod, m, rp, ci, v, rtol=RTOL):
    orp, oci, ov = oracle_mod.assemble(m)
    np.testing.assert_array_equal(rp, orp)
    np.testing.assert_array_equal(ci, oci)
    scale = np.maximum(np.abs(ov), diag_scale(orp, oci, ov))
    assert np.all(np.abs(v - ov) <= rtol * scale)


def _fan(k, closed):
    import meshgen as mg
    n = k if closed else k + 1
    ang = np.linspace(0, 2 * np.pi, n, endpoint=False)
    x = np.concatenate([[0.0], np.cos(ang)])
    y = np.concatenate([[0.0], np.sin(ang)])
    conn = np.array([[0, 1 + i, 1 + (i + 1) % n] for i in range(k)], np.int32)
    conn = np.random.default_rng(k).permutation(conn)
    return mg.Mesh(mg.T3, x, y, None, np.ascontiguousarray(conn), None, None, None, E0=1.0, nu0=0.3)


@pytest.mark.parametrize("k", [3, 7, 8, 9, 12, 13, 14, 15, 16, 125, 126, 127, 200])
@pytest.mark.parametrize("closed", [True, False])
def test_fans(fem, oracle_mod, cuda_device, k, closed):
    m = _fan(k, closed)
    rp, ci, v, info = fem.assemble(m)
    _compare(oracle_mod, m, rp, ci, v)
    cols = k + 1 if closed else k + 2
    assert info["max_row_entries"] == cols
    assert info["overflow_chunks"] == max(0, -(-(cols - 14) // 14))


@pytest.mark.parametrize("nx,ny", [(1, 1), (6, 8), (62, 1), (7, 7), (63, 1), (64, 1), (15, 7), (128, 3)])
@pytest.mark.parametrize("kind", ["q4", "t3", "mixed"])
def test_node_counts_around_a_tile(fem, oracle_mod, cuda_device, kind, nx, ny):
    import meshgen as mg
    m = {"q4": mg.q4_grid, "t3": mg.t3_grid, "mixed": mg.mixed_grid}[kind](nx, ny, seed=nx + ny)
    rp, ci, v, _ = fem.assemble(m)
    _compare(oracle_mod, m, rp, ci, v)


@pytest.mark.parametrize("precision", [0, 3])
def test_repeated_nodes(fem, oracle_mod, cuda_device, precision):
    # quads collapsed to triangles at each of their four positions in turn
    import meshgen as mg
    m = mg.q4_grid(9, 7, seed=3)
    conn = m.conn.copy()
    for e in range(0, conn.shape[0], 3):
        k = (e // 3) % 4
        conn[e, k] = conn[e, (k + 1) % 4]
    m.conn = conn
    rp, ci, v, _ = fem.assemble(m, fem.opts(precision=precision))
    _compare(oracle_mod, m, rp, ci, v, 1e-5 if precision else RTOL)


@pytest.mark.parametrize("off_v,off_c", [(1, 0), (0, 1), (1, 1)])
def test_outputs_off_the_wide_alignment(fem, oracle_mod, cuda_device, off_v, off_c):
    import torch
    import meshgen as mg
    m = mg.by_name("mixed_small")
    a = fem.Assembler(m)
    nnz = int(a.assemble()[3].nnz)
    ci = torch.full((nnz + 2,), -7, dtype=torch.int32, device="cuda")
    v = torch.full((nnz + 2,), 7.0, dtype=torch.float64, device="cuda")
    out = fem.FemCsr(m.num_dofs, 0, 0, nnz, a.row_ptr.data_ptr(), ci[off_c:].data_ptr(), v[off_v:].data_ptr())
    st = fem.load().fem_assemble(C.byref(a.cm), None, C.c_void_p(a.ws_ptr), a.ws_bytes, C.byref(out), None)
    assert st == 0 and out.nnz == nnz
    _compare(oracle_mod, m, a.row_ptr.cpu().numpy(), ci[off_c:off_c + nnz].cpu().numpy(),
             v[off_v:off_v + nnz].cpu().numpy())
    assert v[off_v + nnz].item() == 7.0 and ci[off_c + nnz].item() == -7


def test_batch_of_many_slots_and_unaligned_outputs(fem, oracle_mod, cuda_device):
    # 70 slots: a round of more meshes than one launch's descriptors hold; every
    # third mesh's outputs off the wide alignment (and all kinds in a round)
    import torch
    import meshgen as mg
    meshes = mg.batch_meshes(70, seed=11, emin=1, emax=120)
    b = fem.Batch(meshes, concurrency=70)
    nnz = b.sizes()
    for i in range(0, 70, 3):
        b.col_idx[i] = torch.empty(nnz[i] + 1, dtype=torch.int32, device="cuda")[1:]
        b.values[i] = torch.empty(nnz[i] + 1, dtype=torch.float64, device="cuda")[1:]
    b._set_outs(capacity=True)
    b.run()
    torch.cuda.synchronize()
    assert all(s == 0 for s in b.statuses())
    for i, m in enumerate(meshes):
        _compare(oracle_mod, m, *b.result(i))


@pytest.mark.parametrize("name", ["fan5", "fan13", "fan14", "fan40", "wedge", "q4_7x9", "mixed_33x2", "loose"])
def test_reassembly_rows(fem, oracle_mod, cuda_device, name):
    # rows at the limit of the shared-memory sums (14 columns) and past it,
    # repeated nodes, and mostly unconnected triangles (the block-position map)
    import torch
    import meshgen as mg
    if name.startswith("fan"):
        m = _fan(int(name[3:]), True)
    elif name == "wedge":
        m = mg.q4_grid(9, 7, seed=3)
        conn = m.conn.copy()
        conn[::3, 1] = conn[::3, 2]
        m.conn = conn
    elif name == "loose":
        g = mg.t3_grid(40, 40, seed=2)
        m = mg.Mesh(mg.T3, g.x[g.conn].ravel(), g.y[g.conn].ravel(), None,
                    np.arange(3 * g.num_elems, dtype=np.int32).reshape(-1, 3), None, None, None)
    else:
        m = {"q4_7x9": lambda: mg.q4_grid(7, 9, seed=1), "mixed_33x2": lambda: mg.mixed_grid(33, 2, seed=1)}[name]()
    asm = fem.Assembler(m)
    rp, ci, v, info = asm.assemble()
    re = fem.Reassembler(asm)
    re.build(int(info.nnz))
    vals = torch.full((int(info.nnz) + 1,), 7.0, dtype=torch.float64, device="cuda")
    for _ in range(2):
        re.reassemble(vals)
        assert re.read_info() == 0
        _compare(oracle_mod, m, rp.cpu().numpy(), ci.cpu().numpy(), vals[:-1].cpu().numpy())
        assert vals[-1].item() == 7.0


@pytest.mark.parametrize("name", ["fan5", "fan13", "fan14", "fan40", "wedge", "mixed", "q4_89", "q4_90", "t3_180", "t3_181"])
def test_reassembly_rows_larger(fem, oracle_mod, cuda_device, name):
    # the map by row nodes starts at 8,192 nodes (Q4) and 32,768 (T3, mixed): grids on both sides of the line, and odd
    # pieces beside a grid past it
    import torch
    import meshgen as mg

    def beside(m, g):
        g.conn = np.ascontiguousarray(np.concatenate([g.conn, m.conn + g.num_nodes]).astype(np.int32))
        return mg.Mesh(m.kind, np.concatenate([g.x, m.x + 10.0]), np.concatenate([g.y, m.y]), None, g.conn, None, None,
                       None, E0=1.0, nu0=0.3)

    if name.startswith("fan"):
        m = beside(_fan(int(name[3:]), True), mg.t3_grid(185, 185, seed=2))
    elif name == "wedge":
        w = mg.q4_grid(9, 7, seed=3)
        w.conn = w.conn.copy()
        w.conn[::3, 1] = w.conn[::3, 2]
        m = beside(w, mg.q4_grid(95, 95, seed=2))
    elif name == "mixed":
        m = mg.mixed_grid(200, 180, seed=1)
    else:
        k, n = name.split("_")
        m = (mg.q4_grid if k == "q4" else mg.t3_grid)(int(n), int(n), seed=4)
    asm = fem.Assembler(m)
    rp, ci, v, info = asm.assemble()
    re = fem.Reassembler(asm)
    re.build(int(info.nnz))
    vals = torch.full((int(info.nnz) + 1,), 7.0, dtype=torch.float64, device="cuda")
    for _ in range(2):
        re.reassemble(vals)
        assert re.read_info() == 0
        _compare(oracle_mod, m, rp.cpu().numpy(), ci.cpu().numpy(), vals[:-1].cpu().numpy())
        assert vals[-1].item() == 7.0
