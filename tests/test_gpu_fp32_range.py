"""FP32 blocks of 2-D elements (FEM_PREC_FP32) far from unit size, through the C
ABI: the plane-stress matrix does not depend on the size of the mesh, so meshes
scaled down to element sizes of 1e-17 with a steel-like modulus assemble and
re-assemble within the FP32 form's 1e-5 of max(|K_ij|, sqrt(|K_ii K_jj|)) of the
oracle's matrix of the unscaled mesh (the oracle, like the reference, clamps a
quadrilateral's detJ at a fixed value)."""
import numpy as np
import pytest

from conftest import diag_scale

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nx,ny", [("q4", 12, 9), ("t3", 12, 9), ("mixed", 12, 9), ("q4", 95, 91), ("t3", 185, 181),
                                        ("mixed", 185, 181)])
@pytest.mark.parametrize("scale", [1e-15, 1e-9, 1e9])
def test_sizes(fem, oracle_mod, cuda_device, kind, nx, ny, scale):
    import torch
    import meshgen as mg
    m = {"q4": mg.q4_grid, "t3": mg.t3_grid, "mixed": mg.mixed_grid}[kind](nx, ny, seed=3)
    h = max(nx, ny) / 12  # the larger meshes' elements the size of the smaller ones'
    m.E = m.nu = None
    m.E0, m.nu0 = 2.1e11, 0.3
    orp, oci, ov = oracle_mod.assemble(m)
    m.x, m.y = m.x * scale * h, m.y * scale * h
    o = fem.opts(precision=fem.FEM_PREC_FP32)
    asm = fem.Assembler(m, o)
    rp, ci, v, info = asm.assemble()
    np.testing.assert_array_equal(ci.cpu().numpy(), oci)
    most = 1e-5 * np.maximum(np.abs(ov), diag_scale(orp, oci, ov))
    assert np.all(np.abs(v.cpu().numpy() - ov) <= most)
    re = fem.Reassembler(asm)
    re.build(int(info.nnz))
    vals = torch.full((int(info.nnz),), 7.0, dtype=torch.float64, device="cuda")
    re.reassemble(vals, o)
    assert re.read_info() == 0
    assert np.all(np.abs(vals.cpu().numpy() - ov) <= most)


def test_t3_blocks_that_fp32_holds(fem, oracle_mod, cuda_device):
    # integer coordinates, nu = 0, thickness 2 and E = detJ: every factor and sum of a block is a whole number or a half
    # below 2^24, so the FP32 form has no rounding to make (what is left is the oracle's: 1e-12, as in FP64)
    import torch
    import meshgen as mg
    nx, ny = 185, 181
    m = mg.t3_grid(nx, ny, seed=3)
    r = np.random.default_rng(3)
    at = np.arange(m.num_nodes)
    m.x = 32.0 * (at % (nx + 1)) + r.integers(-7, 8, m.num_nodes)
    m.y = 32.0 * (at // (nx + 1)) + r.integers(-7, 8, m.num_nodes)
    x, y = m.x[m.conn], m.y[m.conn]
    m.E = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (x[:, 2] - x[:, 0]) * (y[:, 1] - y[:, 0])
    assert m.E.min() > 0
    m.nu, m.nu0, m.thickness = None, 0.0, 2.0
    orp, oci, ov = oracle_mod.assemble(m)
    o = fem.opts(precision=fem.FEM_PREC_FP32)
    asm = fem.Assembler(m, o)
    rp, ci, v, info = asm.assemble()
    np.testing.assert_array_equal(ci.cpu().numpy(), oci)
    most = 1e-12 * np.maximum(np.abs(ov), diag_scale(orp, oci, ov))
    assert np.all(np.abs(v.cpu().numpy() - ov) <= most)
    re = fem.Reassembler(asm)
    re.build(int(info.nnz))
    re.reassemble(v, o)
    assert re.read_info() == 0
    assert np.all(np.abs(v.cpu().numpy() - ov) <= most)
