"""What a scatter map takes in (fem_scatter_map_build, fem_reassemble_values),
through the C ABI: elements with a bad node id, in both forms of the map (by
element blocks, small 2-D meshes and Hex20; by row nodes, larger 2-D meshes).
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
