"""What a scatter map takes in (fem_scatter_map_build, fem_reassemble_values),
through the C ABI: elements with a bad node id, and a caller's own patterns
(further columns and rows, missing blocks, a row of more than 65,536 columns), in
both forms of the map (by element blocks, small 2-D meshes and Hex20; by row
nodes, larger 2-D meshes).
Values within 1e-12 of max(|K_ij|, sqrt(|K_ii K_jj|)) of the oracle's assembly."""
import copy

import numpy as np
import pytest

from conftest import diag_scale

pytestmark = pytest.mark.gpu

RTOL = 1e-12
# meshes on both sides of the line from which the map of a 2-D mesh is by row nodes (8,192 nodes Q4, 32,768 T3 and mixed)
MESHES = {"q4_small": ("q4_grid", 12, 9), "t3_small": ("t3_grid", 12, 9), "mixed_small": ("mixed_grid", 12, 9),
          "q4_large": ("q4_grid", 95, 91), "t3_large": ("t3_grid", 185, 181), "mixed_large": ("mixed_grid", 185, 181)}


def _mesh(name):
    import meshgen as mg
    f, nx, ny = MESHES[name]
    return getattr(mg, f)(nx, ny, seed=7)


def _close(orp, oci, ov, got):
    scale = np.maximum(np.abs(ov), diag_scale(orp, oci, ov))
    assert np.all(np.abs(got - ov) <= RTOL * scale)


def _build(fem, asm, nnz, status):
    """A Reassembler whose map build ends with `status`."""
    re = fem.Reassembler(asm)
    try:
        re.build(nnz)
        assert status == 0
    except fem.FemError as e:
        assert e.status == status
    return re


@pytest.mark.parametrize("name", list(MESHES) + ["hex20"])
def test_elements_with_a_bad_node_take_no_part(fem, oracle_mod, cuda_device, name):
    # the pattern of the whole mesh; then elements get a bad id at each position in turn (the id past the last node, and -1)
    import torch
    import meshgen as mg
    m = mg.hex20_grid(3, 3, 2, seed=7) if name == "hex20" else _mesh(name)
    asm = fem.Assembler(m)
    rp, ci, v, info = asm.assemble()
    nnz = int(info.nnz)
    orp, oci, _ = oracle_mod.assemble(m)
    bad = np.arange(0, m.num_elems, 5)
    npe = 20 if name == "hex20" else (np.where(m.types[bad] == mg.Q4, 4, 3) if m.types is not None else m.conn.shape[1])
    at = np.arange(bad.size) % npe
    asm.dev["conn"][torch.from_numpy(bad).cuda(), torch.from_numpy(at).cuda()] = torch.from_numpy(
        np.where(np.arange(bad.size) % 2 == 0, m.num_nodes, -1).astype(np.int32)).cuda()
    re = _build(fem, asm, nnz, fem.FEM_ERR_BAD_MESH)
    vals = torch.full((nnz,), 7.0, dtype=torch.float64, device="cuda")
    re.reassemble(vals)
    m2 = copy.copy(m)
    m2.E = np.array(m.E if m.E is not None else np.full(m.num_elems, m.E0))
    m2.nu = np.array(m.nu if m.nu is not None else np.full(m.num_elems, m.nu0))
    full = oracle_mod.assemble(m2)[2]
    m2.E[bad] = 0.0
    ov = oracle_mod.assemble(m2)[2]
    scale = np.maximum(np.abs(full), diag_scale(orp, oci, full))
    assert np.all(np.abs(vals.cpu().numpy() - ov) <= RTOL * scale)


def _extended(rp, ci, lead, tail, rows):
    """The pattern (rp, ci) with `lead` further columns in front of every row, `tail` behind it (the columns move up by
    `lead`) and `rows` further rows of one entry at the end; and where each old entry went."""
    n = rp.size - 1
    length = np.diff(rp)
    rp2 = np.concatenate([[0], np.cumsum(length + lead + tail), rp[-1] + n * (lead + tail) + 1 + np.arange(rows)])
    ci2 = np.zeros(rp2[-1], np.int32)
    at = np.repeat(rp2[:n] + lead - rp[:-1], length) + np.arange(rp[-1])
    ci2[at] = ci
    for k in range(lead):
        ci2[rp2[:n] + k] = k - lead
    for k in range(tail):
        ci2[rp2[1:n + 1] - tail + k] = n + k
    return rp2.astype(np.int32), ci2, at


def _with_pattern(asm, rp, ci):
    import torch
    asm.row_ptr = torch.from_numpy(np.ascontiguousarray(rp, np.int32)).cuda()
    asm.col_idx = torch.from_numpy(np.ascontiguousarray(ci, np.int32)).cuda()
    return torch.full((ci.size,), 7.0, dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("name", list(MESHES))
@pytest.mark.parametrize("lead,tail,rows", [(0, 1, 1), (1, 0, 0), (2, 1, 0), (2, 0, 3), (0, 2, 2)])
def test_patterns_with_further_entries(fem, oracle_mod, cuda_device, name, lead, tail, rows):
    # the mesh's entries get the assembled values, all others are zero
    m = _mesh(name)
    orp, oci, ov = oracle_mod.assemble(m)
    rp, ci, at = _extended(orp, oci, lead, tail, rows)
    asm = fem.Assembler(m)
    vals = _with_pattern(asm, rp, ci)
    re = _build(fem, asm, ci.size, 0)
    for _ in range(2):
        vals.fill_(7.0)
        re.reassemble(vals)
        assert re.read_info() == 0
        got = vals.cpu().numpy()
        _close(orp, oci, ov, got[at])
        assert np.all(np.delete(got, at) == 0.0)


@pytest.mark.parametrize("name", list(MESHES))
def test_patterns_without_some_blocks(fem, oracle_mod, cuda_device, name):
    # the last column node of every 50th row node left out: reported when the map is built, the others are right
    m = _mesh(name)
    orp, oci, ov = oracle_mod.assemble(m)
    keep = np.ones(oci.size, bool)
    nodes = np.arange(0, m.num_nodes, 50)
    for r in (2 * nodes, 2 * nodes + 1):
        keep[orp[r + 1] - 1] = keep[orp[r + 1] - 2] = False
    rp = np.concatenate([[0], np.cumsum(keep)[orp[1:] - 1]])
    asm = fem.Assembler(m)
    vals = _with_pattern(asm, rp, oci[keep])
    re = _build(fem, asm, int(keep.sum()), fem.FEM_ERR_INTERNAL)
    re.reassemble(vals)
    scale = np.maximum(np.abs(ov), diag_scale(orp, oci, ov))
    assert np.all(np.abs(vals.cpu().numpy() - ov[keep]) <= RTOL * scale[keep])


@pytest.mark.parametrize("name", list(MESHES))
@pytest.mark.parametrize("first", [1, 2, 7])
def test_patterns_that_start_behind_other_entries(fem, oracle_mod, cuda_device, name, first):
    # the rows of one matrix among others: row_ptr[0] is not 0; the entries before it become zero, as those behind the rows
    m = _mesh(name)
    orp, oci, ov = oracle_mod.assemble(m)
    asm = fem.Assembler(m)
    vals = _with_pattern(asm, orp + first, np.concatenate([np.zeros(first, np.int32), oci]))
    re = _build(fem, asm, vals.numel(), 0)
    re.reassemble(vals)
    assert re.read_info() == 0
    got = vals.cpu().numpy()
    assert np.all(got[:first] == 0.0)
    _close(orp, oci, ov, got[first:])


@pytest.mark.parametrize("cols", [65535, 65536, 65537, 70001])
def test_rows_past_16_bit_ranks(fem, oracle_mod, cuda_device, cols):
    # a closed fan: its hub's row has a column per triangle and its own
    import meshgen as mg
    k = cols - 1
    ang = np.linspace(0, 2 * np.pi, k, endpoint=False)
    conn = np.stack([np.full(k, k // 2), np.arange(k), (np.arange(k) + 1) % k], 1)
    conn[:, 1:] += conn[:, 1:] >= k // 2  # the hub's id in the middle
    xy = np.insert(np.stack([np.cos(ang), np.sin(ang)], 1), k // 2, 0.0, axis=0)
    conn = np.random.default_rng(1).permutation(conn).astype(np.int32)
    m = mg.Mesh(mg.T3, xy[:, 0].copy(), xy[:, 1].copy(), None, np.ascontiguousarray(conn), None, None, None, E0=1.0, nu0=0.3)
    rp, ci, v = oracle_mod.assemble(m)
    assert np.diff(rp).max() == 2 * cols
    asm = fem.Assembler(m)
    vals = _with_pattern(asm, rp, ci)
    re = _build(fem, asm, ci.size, 0)
    re.reassemble(vals)
    assert re.read_info() == 0
    # the hub's entries are sums of up to 70,001 terms: 1e-10 of its diagonal covers their order
    scale = np.maximum(np.abs(v), diag_scale(rp, ci, v))
    assert np.all(np.abs(vals.cpu().numpy() - v) <= 1e-10 * scale)


# columns that a thread sums in shared memory: 10 (T3), 14 (Q4, mixed); longer rows are added with atomics
@pytest.mark.parametrize("kind,k", [("t3", 8), ("t3", 9), ("t3", 10), ("t3", 40), ("q4", 6), ("q4", 7), ("q4", 30), ("mixed", 6),
                                    ("mixed", 7), ("mixed", 30)])
@pytest.mark.parametrize("precision", [0, 3])
def test_rows_around_the_sums_of_a_thread(fem, oracle_mod, cuda_device, kind, k, precision):
    # fans of k triangles (k + 1 columns) or quadrilaterals (2 k + 1), one beside another and a grid by row nodes
    import torch
    import meshgen as mg
    from test_gpu_hubs import _beside, _mixed_fan, _quad_fan, _shuffled
    from test_gpu_rows2d import _fan
    fan = {"t3": lambda: _shuffled(_fan(k, True)), "q4": lambda: _quad_fan(k), "mixed": lambda: _mixed_fan(k)}[kind]
    g = _mesh(kind + "_large")
    g.E = g.nu = None
    m = _beside(fan(), _beside(fan(), g))
    asm = fem.Assembler(m)
    rp, ci, v, info = asm.assemble()
    re = _build(fem, asm, int(info.nnz), 0)
    vals = torch.full((int(info.nnz),), 7.0, dtype=torch.float64, device="cuda")
    re.reassemble(vals, fem.opts(precision=precision))
    assert re.read_info() == 0
    orp, oci, ov = oracle_mod.assemble(m)
    scale = np.maximum(np.abs(ov), diag_scale(orp, oci, ov))
    assert np.all(np.abs(vals.cpu().numpy() - ov) <= (1e-5 if precision else RTOL) * scale)
