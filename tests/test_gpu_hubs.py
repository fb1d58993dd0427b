"""Nodes with far more elements or columns than those of a regular mesh, through
the C ABI against the oracle, alone (small meshes: one cooperative launch) and
beside a grid of more than 16,384 nodes (a launch per phase; Hex20: a node
order). Full, block and upper-triangle output. Pattern bit for bit; values
within 1e-12 plus the rounding of two sums of `terms` entries, 2 terms 2^-52, of
max(|K_ij|, sqrt(|K_ii K_jj|))."""
import numpy as np
import pytest

from conftest import diag_scale
from test_gpu_rows_hex20 import _copies, _star

pytestmark = pytest.mark.gpu


def _beside(m, g):
    """The mesh m moved away from the grid g, one mesh of both."""
    import meshgen as mg
    conn = np.ascontiguousarray(np.concatenate([g.conn, m.conn + g.num_nodes]).astype(np.int32))
    types = None if m.types is None else np.concatenate([g.types, m.types])
    z = None if m.z is None else np.concatenate([g.z, m.z])
    E = None if m.E is None else np.concatenate([np.ones(g.num_elems), m.E])
    nu = None if E is None else np.full(conn.shape[0], 0.3)
    return mg.Mesh(m.kind, np.concatenate([g.x, m.x + 10.0]), np.concatenate([g.y, m.y]), z, conn, types, E, nu, E0=1.0, nu0=0.3)


def _check(fem, oracle_mod, m, terms, o=None, forms=True):
    rtol = 1e-12 + 2 * terms * 2.0 ** -52
    asm = fem.Assembler(m, o)
    rp, ci, v, info = asm.assemble()
    rp, ci, v = rp.cpu().numpy(), ci.cpu().numpy(), v.cpu().numpy()
    orp, oci, ov = oracle_mod.assemble(m)
    np.testing.assert_array_equal(rp, orp)
    np.testing.assert_array_equal(ci, oci)
    assert np.all(np.abs(v - ov) <= rtol * np.maximum(np.abs(ov), diag_scale(orp, oci, ov)))
    if not forms:
        return info
    d = m.dpn
    brp, bci, bv = (t.cpu().numpy() for t in asm.consolidate_bsr())
    np.testing.assert_array_equal(brp * d * d, orp[::d])
    at = np.repeat(orp[:-1:d], np.diff(brp)) + d * (np.arange(bci.shape[0]) - np.repeat(brp[:-1], np.diff(brp)))
    np.testing.assert_array_equal(bci * d, oci[at])
    u = np.repeat(d * np.diff(brp), np.diff(brp))
    for i in range(d):
        for j in range(d):
            np.testing.assert_array_equal(bv.reshape(-1, d * d)[:, d * i + j], v[at + i * u + j])
    urp, uci, uv = (t.cpu().numpy() for t in asm.consolidate_upper())
    keep = oci >= np.repeat(np.arange(m.num_dofs), np.diff(orp))
    assert urp[-1] == keep.sum()
    np.testing.assert_array_equal(uci, oci[keep])
    np.testing.assert_array_equal(uv, v[keep])
    return info


# Hex20: 204 elements have 4,080 candidate columns, one stretch of the sort; 205 need several
@pytest.mark.parametrize("k", [33, 34, 204, 205, 300])
@pytest.mark.parametrize("beside", [False, True])
def test_hex20_stars(fem, oracle_mod, cuda_device, k, beside):
    import meshgen as mg
    m = _star(k)
    if beside:
        m = _beside(m, mg.hex20_grid(17, 17, 17, seed=3))
    info = _check(fem, oracle_mod, m, k)
    assert info.overflow_chunks == -(-(1 + 19 * k - 94) // 30)
    assert info.max_row_entries == 1 + 19 * k


@pytest.mark.parametrize("k", [5, 60, 520])
@pytest.mark.parametrize("beside", [False, True])
def test_hex20_copies(fem, oracle_mod, cuda_device, k, beside):
    # 8 k elements at the middle node; at 520 its own id alone is more than a stretch
    import meshgen as mg
    m = _copies(k)
    if beside:
        m = _beside(m, mg.hex20_grid(17, 17, 17, seed=3))
    _check(fem, oracle_mod, m, 8 * k)


@pytest.mark.parametrize("k", [120, 250])
def test_hex20_star_that_overflows_the_pool(fem, cuda_device, k):
    # more columns than the 46 + 65 * 30 of a first chunk and the whole pool: the row is cut and the status says so
    m = _star(k)
    with pytest.raises(fem.FemError) as e:
        fem.assemble(m, fem.opts(first_slots=46, pool_factor=1e-9))
    assert e.value.status == fem.FEM_ERR_POOL_OVERFLOW


# 3,449 elements: 65,532 columns; 3,450: 65,551, past the 65,536 that the rank map numbers
@pytest.mark.parametrize("k", [3449, 3450])
def test_hex20_rows_past_16_bit_ranks(fem, oracle_mod, cuda_device, k):
    _check(fem, oracle_mod, _star(k), k, forms=False)


def _quad_fan(k):
    """k quadrilaterals around one node (2 k + 1 columns in its row), node ids shuffled."""
    import meshgen as mg
    ang = np.linspace(0, 2 * np.pi, 2 * k, endpoint=False)
    r = np.where(np.arange(2 * k) % 2 == 0, 1.0, 1.0 / np.cos(np.pi / (2 * k)))  # the quads stay convex
    x, y = np.concatenate([[0.0], r * np.cos(ang)]), np.concatenate([[0.0], r * np.sin(ang)])
    i = np.arange(k)
    conn = np.stack([np.zeros(k, int), 1 + 2 * i, 2 + 2 * i, 1 + (2 * i + 2) % (2 * k)], 1)
    return _shuffled(mg.Mesh(mg.Q4, x, y, None, conn, None, None, None, E0=1.0, nu0=0.3))


def _book(k):
    """k triangles on one common edge: two hubs, the list of further elements (2 (k - 126) of them) longer than k from k = 253 on."""
    import meshgen as mg
    x = np.concatenate([[0.0, 1.0], np.linspace(0.1, 0.9, k)])
    y = np.concatenate([[0.0, 0.0], 1.0 + 0.1 * np.sin(np.arange(k))])
    conn = np.stack([np.zeros(k, int), np.ones(k, int), 2 + np.arange(k)], 1)
    conn = np.stack([np.roll(c, s) for s, c in zip(np.arange(k) % 3, conn)])
    return _shuffled(mg.Mesh(mg.T3, x, y, None, conn, None, None, None, E0=1.0, nu0=0.3))


def _mixed_fan(k):
    """A fan of k triangles whose every other element is a quadrilateral of two neighbouring rim edges."""
    import meshgen as mg
    m = _quad_fan(k)
    m.kind = mg.MIXED_2D
    m.types = np.where(np.arange(k) % 2 == 0, mg.Q4, mg.T3).astype(np.uint8)
    return m


def _shuffled(m):
    rng = np.random.default_rng(m.num_elems)
    p = rng.permutation(m.num_nodes)
    inv = np.argsort(p)
    m.x, m.y = m.x[inv], m.y[inv]
    m.conn = np.ascontiguousarray(rng.permutation(p[m.conn]).astype(np.int32))
    return m


# a row's own storage keeps 126 elements; a CTA takes 64 at a time and searches the further ones 1,024 at a time
@pytest.mark.parametrize("name,k", [("t3", 126), ("t3", 127), ("t3", 360), ("t3", 1150), ("t3", 1151), ("t3", 2300),
                                    ("q4", 63), ("q4", 126), ("q4", 127), ("q4", 400), ("mixed", 126), ("mixed", 300),
                                    ("book", 126), ("book", 127), ("book", 252), ("book", 253), ("book", 1500)])
@pytest.mark.parametrize("beside", [False, True])
def test_2d_hubs(fem, oracle_mod, cuda_device, name, k, beside):
    import meshgen as mg
    from test_gpu_rows2d import _fan
    m = {"t3": lambda: _shuffled(_fan(k, True)), "q4": lambda: _quad_fan(k), "mixed": lambda: _mixed_fan(k),
         "book": lambda: _book(k)}[name]()
    if beside:
        g = {"q4": mg.q4_grid, "mixed": mg.mixed_grid}.get(name, mg.t3_grid)(131, 130, seed=5)
        g.E = g.nu = None
        m = _beside(m, g)
    info = _check(fem, oracle_mod, m, k, fem.opts(pool_factor=1.0))
    if not beside:
        rows = np.diff(oracle_mod.pattern(m)[0])[::2] // 2
        assert info.overflow_chunks == np.maximum(0, -(-(rows - 14) // 14)).sum()


def test_2d_hubs_that_share_elements_and_many_of_them(fem, oracle_mod, cuda_device):
    # fans of different sizes beside one another: their further elements share one list
    from test_gpu_rows2d import _fan
    m = _fan(130, True)
    for k in (127, 500, 14, 200, 360):
        m = _beside(_fan(k, k != 200), m)
    _check(fem, oracle_mod, m, 500, fem.opts(pool_factor=1.0))
