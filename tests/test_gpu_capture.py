"""Single-mesh calls captured in a CUDA graph and on two streams at a time, through
the C ABI: small meshes, whose lists one cooperative launch builds, and larger
ones. Values within 1e-12 of max(|K_ij|, sqrt(|K_ii K_jj|)) of the oracle."""
import threading

import numpy as np
import pytest

from conftest import diag_scale

pytestmark = pytest.mark.gpu

MESHES = ["q4_small", "t3_small", "mixed_small", "hex20_small", "t3_large", "q4_large", "hex20_large"]


def _mesh(name):
    import meshgen as mg
    return {"q4_small": lambda: mg.q4_grid(12, 9, seed=3), "t3_small": lambda: mg.t3_grid(12, 9, seed=3),
            "mixed_small": lambda: mg.mixed_grid(12, 9, seed=3), "hex20_small": lambda: mg.hex20_grid(4, seed=3),
            "t3_large": lambda: mg.t3_grid(185, 181, seed=3), "q4_large": lambda: mg.q4_grid(131, 130, seed=3),
            "hex20_large": lambda: mg.hex20_grid(17, seed=3)}[name]()


def _close(ref, asm, values=None):
    orp, oci, ov = ref
    n = oci.size
    np.testing.assert_array_equal(asm.row_ptr.cpu().numpy(), orp)
    np.testing.assert_array_equal(asm.col_idx[:n].cpu().numpy(), oci)
    got = (asm.values if values is None else values)[:n].cpu().numpy()
    assert np.all(np.abs(got - ov) <= 1e-12 * np.maximum(np.abs(ov), diag_scale(orp, oci, ov)))


@pytest.mark.parametrize("name", MESHES)
def test_in_a_graph(fem, oracle_mod, cuda_device, name):
    import torch
    m = _mesh(name)
    asm = fem.Assembler(m)
    nnz = int(asm.assemble()[3].nnz)
    re = fem.Reassembler(asm)
    re.build(nnz)
    vals = torch.empty(nnz, dtype=torch.float64, device="cuda")
    re.reassemble(vals)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        asm.assemble_async()
        re.reassemble(vals)
    ref = oracle_mod.assemble(m)
    for _ in range(2):
        asm.row_ptr.zero_()
        asm.col_idx.zero_()
        asm.values.zero_()
        vals.fill_(7.0)
        g.replay()
        torch.cuda.synchronize()
        assert asm.read_info()[0] == 0 and re.read_info() == 0
        _close(ref, asm)
        _close(ref, asm, vals)


@pytest.mark.parametrize("first,second", [("q4_small", "q4_small"), ("t3_small", "hex20_small"), ("mixed_small", "t3_large"),
                                          ("hex20_small", "hex20_large")])
def test_on_two_streams(fem, oracle_mod, cuda_device, first, second):
    import torch
    meshes = [_mesh(first), _mesh(second)]
    asms = [fem.Assembler(m) for m in meshes]
    for a in asms:
        a.assemble()
    refs = [oracle_mod.assemble(m) for m in meshes]
    torch.cuda.synchronize()
    errors = []

    def work(a):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(50):
                    a.assemble_async()
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(a,)) for a in asms]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for a, ref in zip(asms, refs):
        assert a.read_info()[0] == 0
        _close(ref, a)
