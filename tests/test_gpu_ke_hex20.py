"""The one-warp-per-element FP64 Hex20 Ke kernel (ke_hex20.cu) at element counts
around a CTA's warps, with a bad element between good ones and with an output
that is not 16-byte aligned (plain stores instead of the bulk copy), against
the oracle within 1e-12 of the element's largest diagonal entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(fem, oracle_mod, m, ke, skip=()):
    ke = ke.cpu().numpy()
    for e in range(m.num_elems):
        if e in skip:
            assert np.all(ke[e] == 0.0)
            continue
        n = m.conn[e]
        E, nu = (m.E[e], m.nu[e]) if m.E is not None else (m.E0, m.nu0)
        ref = oracle_mod.ke_hex20(m.x[n], m.y[n], m.z[n], E, nu)
        got = fem.unpack_element_stiffness(ke[e], 20, 3)
        assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(np.diag(ref))), e


def _mesh(count, seed=5):
    import meshgen as mg
    m = mg.hex20_grid(5, 4, 2, seed=seed)
    m.conn = m.conn[:count].copy()
    r = np.random.default_rng(seed)
    m.E, m.nu = r.lognormal(0, 0.5, count), r.uniform(0.1, 0.45, count)
    return m


@pytest.mark.parametrize("count", [1, 7, 8, 9, 17, 40])
@pytest.mark.parametrize("offset", [0, 1])
def test_counts_and_alignment(fem, oracle_mod, cuda_device, count, offset):
    import torch
    m = _mesh(count)
    buf = torch.full((count * 1890 + 2,), 7.0, dtype=torch.float64, device="cuda")
    out = buf[offset:offset + count * 1890].view(count, 1890)
    ke, status = fem.element_stiffness(m, out=out)
    assert status == 0
    _check(fem, oracle_mod, m, ke)
    assert buf[offset + count * 1890].item() == 7.0


@pytest.mark.parametrize("bad", [[0], [3, 4], [8], [16]])
def test_bad_elements_between_good_ones(fem, oracle_mod, cuda_device, bad):
    m = _mesh(17)
    for k, e in enumerate(bad):
        m.conn[e, 3 * k] = m.num_nodes if k % 2 == 0 else -1
    ke, status = fem.element_stiffness(m)
    assert status == 1 << fem.FEM_ERR_BAD_MESH
    _check(fem, oracle_mod, m, ke, skip=bad)
