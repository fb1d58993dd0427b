"""The Hex20 row lists (rows_hex20.cu) and their gather (write_hex20.cu) at the
sizes where they change path, through the C ABI against the oracle: nodes with
up to 8, 9 to 32 and more elements; rows past the first chunk, past the
gather's window of 96 columns and past 256; elements with repeated nodes; full,
block and upper-triangle output. Pattern bit for bit, values within 1e-12 of
max(|K_ij|, sqrt(|K_ii K_jj|))."""
import numpy as np
import pytest

from conftest import diag_scale

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def _star(k):
    """k unit cubes that share one corner node and nothing else."""
    import meshgen as mg
    one = mg.hex20_grid(1, jitter=0.0)
    conn = np.empty((k, 20), np.int32)
    x, y, z = ([c[one.conn[0, 0]]] for c in (one.x, one.y, one.z))
    for e in range(k):
        conn[e, 0] = 0
        for a in range(1, 20):
            conn[e, a] = len(x)
            n = one.conn[0, a]
            s = 1.0 + 0.01 * e
            x.append(one.x[n] * s)
            y.append(one.y[n] * s)
            z.append(one.z[n] * s)
    p = np.random.default_rng(k).permutation(len(x)).astype(np.int32)
    inv = np.argsort(p)
    return mg.Mesh(mg.HEX20, np.array(x)[inv], np.array(y)[inv], np.array(z)[inv], np.ascontiguousarray(p[conn]), None,
                   None, None, E0=1.0, nu0=0.3)


def _copies(k):
    """A 2x2x2 grid with every element k times (own materials): many elements, few columns."""
    import meshgen as mg
    m = mg.hex20_grid(2, seed=9)
    m.conn = np.ascontiguousarray(np.tile(m.conn, (k, 1)))
    m.E = np.random.default_rng(k).uniform(0.5, 2.0, m.num_elems)
    return m


def _wedges():
    """Every other element's face collapsed to an edge (five repeated nodes)."""
    import meshgen as mg
    m = mg.hex20_grid(3, 2, 2, jitter=0.0, seed=4)
    conn = m.conn.copy()
    for a, b in ((3, 2), (10, 2), (7, 6), (14, 6), (19, 18)):
        conn[::2, a] = conn[::2, b]
    m.conn = conn
    return m


def _check(fem, oracle_mod, m, o=None, allow=(0,)):
    asm = fem.Assembler(m, o)
    rp, ci, v, info = asm.assemble(allow)
    rp, ci, v = rp.cpu().numpy(), ci.cpu().numpy(), v.cpu().numpy()
    orp, oci, ov = oracle_mod.assemble(m)
    np.testing.assert_array_equal(rp, orp)
    np.testing.assert_array_equal(ci, oci)
    scale = np.maximum(np.abs(ov), diag_scale(orp, oci, ov))
    assert np.all(np.abs(v - ov) <= RTOL * scale)
    assert info.list_entries == oci.shape[0] // 9 and info.max_row_entries == np.diff(orp).max() // 3
    brp, bci, bv = (t.cpu().numpy() for t in asm.consolidate_bsr())
    np.testing.assert_array_equal(brp * 9, orp[::3])
    at = np.repeat(orp[:-1:3], np.diff(brp)) + 3 * (np.arange(bci.shape[0]) - np.repeat(brp[:-1], np.diff(brp)))
    np.testing.assert_array_equal(bci * 3, oci[at])
    np.testing.assert_array_equal(bv.reshape(-1, 9)[:, 0], v[at])
    urp, uci, uv = asm.consolidate_upper()
    rows = np.repeat(np.arange(m.num_dofs), np.diff(rp))
    keep = ci >= rows
    assert int(urp[-1]) == keep.sum()
    np.testing.assert_array_equal(uci.cpu().numpy()[:keep.sum()], ci[keep])
    np.testing.assert_array_equal(uv.cpu().numpy()[:keep.sum()], v[keep])
    return info


@pytest.mark.parametrize("k", [1, 4, 5, 8, 9, 13, 14, 32, 33])
def test_star(fem, oracle_mod, cuda_device, k):
    info = _check(fem, oracle_mod, _star(k))
    cols = 1 + 19 * k
    assert info.overflow_chunks == max(0, -(-(cols - 94) // 30))


@pytest.mark.parametrize("k", [1, 2, 4, 5])
def test_copies(fem, oracle_mod, cuda_device, k):
    _check(fem, oracle_mod, _copies(k))


def test_repeated_nodes(fem, oracle_mod, cuda_device):
    _check(fem, oracle_mod, _wedges())
    _check(fem, oracle_mod, _wedges(), fem.opts(first_slots=30, chunk_slots=10, pool_factor=4.0))


@pytest.mark.parametrize("shape", [(1, 1, 1), (7, 1, 1), (5, 3, 2), (8, 8, 8)])
@pytest.mark.parametrize("shuffle", [False, True])
def test_grids(fem, oracle_mod, cuda_device, shape, shuffle):
    import meshgen as mg
    m = mg.hex20_grid(*shape, seed=sum(shape))
    if shuffle:
        r = np.random.default_rng(1)
        m.conn = np.ascontiguousarray(m.conn[r.permutation(m.num_elems)])
        m.E, m.nu = r.lognormal(0, 0.5, m.num_elems), r.uniform(0.2, 0.4, m.num_elems)
    _check(fem, oracle_mod, m)


def test_bad_element_leaves_the_others(fem, oracle_mod, cuda_device):
    # an element with a bad node id takes no part; the rest assembles
    import meshgen as mg
    m = mg.hex20_grid(3, 2, 2, seed=6)
    good = m.conn.copy()
    m.conn = good.copy()
    m.conn[4, 7] = m.num_nodes
    asm = fem.Assembler(m)
    rp, ci, v, info = asm.assemble((fem.FEM_ERR_BAD_MESH,))
    m.conn = np.delete(good, 4, axis=0)
    asm.reserve(400 * 9 * 12)
    asm.consolidate()
    st, info = asm.read_info()
    assert st == fem.FEM_ERR_BAD_MESH
    n = int(info.nnz)
    orp, oci, ov = oracle_mod.assemble(m)
    np.testing.assert_array_equal(asm.row_ptr.cpu().numpy(), orp)
    np.testing.assert_array_equal(asm.col_idx[:n].cpu().numpy(), oci)
    scale = np.maximum(np.abs(ov), diag_scale(orp, oci, ov))
    assert np.all(np.abs(asm.values[:n].cpu().numpy() - ov) <= RTOL * scale)


@pytest.mark.parametrize("name", ["grid", "star4", "star5", "star8", "wedges"])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_connectivity_alignment(fem, oracle_mod, cuda_device, name, offset):
    # node ids are read four or two at a time when conn is 16-byte aligned; nodes of up to 4 elements take eight
    # lanes an element and half the table, nodes of 5 to 8 four lanes and the whole one
    import torch
    import meshgen as mg
    m = mg.hex20_grid(4, 3, 3, seed=6) if name == "grid" else _wedges() if name == "wedges" else _star(int(name[4:]))
    asm = fem.Assembler(m)
    buf = torch.empty(m.conn.size + 4, dtype=torch.int32, device="cuda")
    conn = buf[offset:offset + m.conn.size]
    conn.copy_(torch.from_numpy(m.conn.ravel()))
    asm.cm.conn = conn.data_ptr()
    rp, ci, v, info = asm.assemble()
    orp, oci, ov = oracle_mod.assemble(m)
    rp, ci, v = rp.cpu().numpy(), ci.cpu().numpy()[:len(oci)], v.cpu().numpy()[:len(oci)]
    np.testing.assert_array_equal(rp, orp)
    np.testing.assert_array_equal(ci, oci)
    sc = diag_scale(orp, oci, ov)
    assert np.all(np.abs(v - ov) <= RTOL * np.maximum(np.abs(ov), sc))
