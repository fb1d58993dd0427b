"""What the consolidation writes when its output does not fit, or its lists are
not those of the mesh, through the C ABI: nothing outside the caller's buffers,
and a status that says so. The lists' row counts (and list words) are changed in
the workspace between the scatter and the consolidation."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(kind):
    import meshgen as mg
    return {"q4": lambda: mg.q4_grid(9, 7, seed=2), "t3": lambda: mg.t3_grid(9, 7, seed=2),
            "hex20": lambda: mg.hex20_grid(3, 2, 2, seed=2),
            "hex20_ordered": lambda: mg.hex20_grid(15, 15, 15, seed=2)}[kind]()


def _row_counts(torch, asm, rp):
    """The workspace's count array (columns per row node), found by its contents."""
    dpn = asm.mesh.dpn
    want = ((rp[1::dpn] - rp[:-1:dpn]) // dpn).to(torch.int32)
    first = asm.ws_ptr - asm.ws.data_ptr()
    words = asm.ws[first:first + asm.ws_bytes // 4 * 4].view(torch.int32)
    n = want.numel()
    at = torch.nonzero((words[:-n] == want[0]) & (words[n - 1:-1] == want[-1])).flatten().tolist()
    hits = [i for i in at if torch.equal(words[i:i + n], want)]
    assert len(hits) == 1, hits
    return words[hits[0]:hits[0] + n]


@pytest.mark.parametrize("kind", ["q4", "t3", "hex20", "hex20_ordered"])
@pytest.mark.parametrize("form", ["csr", "bsr", "csr_unaligned"])
def test_entries_past_int32_are_not_written(fem, cuda_device, kind, form):
    # counts that add up to more than 2^31 entries (BSR: blocks), and a capacity that promises room for them: the row
    # pointers wrap, so nothing may be stored (the buffers hold 64 entries)
    import torch
    m = _mesh(kind)
    asm = fem.Assembler(m)
    asm.ws.zero_()
    rp = asm.assemble()[0]
    counts = _row_counts(torch, asm, rp)
    counts.fill_(3 * 2 ** 31 // m.num_nodes)
    ci = torch.full((80,), -7, dtype=torch.int32, device="cuda")
    v = torch.full((80,), 7.0, dtype=torch.float64, device="cuda")
    off = 1 if form == "csr_unaligned" else 0
    call = asm.lib.fem_alls_consolidate_bsr if form == "bsr" else asm.lib.fem_alls_consolidate
    st = call(C.byref(asm.cm), C.byref(asm.opts), asm.ws_ptr, asm.ws_bytes, asm.row_ptr.data_ptr(),
              ci[off:].data_ptr(), v[off:].data_ptr(), 2 ** 40, asm._stream())
    assert st == 0
    st, info = asm.read_info()
    assert st == fem.FEM_ERR_RANGE
    assert info.nnz > 2 ** 31
    assert torch.all(ci == -7).item() and torch.all(v == 7.0).item()


def _slots(torch, asm):
    """The first chunks' rows in the workspace (behind the info word): [nodes, 2 + slots] words."""
    h = 96 if asm.mesh.dpn == 3 else 16
    first = asm.ws_ptr - asm.ws.data_ptr() + 256
    n = asm.mesh.num_nodes
    return asm.ws[first:first + n * h * 4].view(torch.int32).view(n, h)


def _consolidate(asm, form, nnz):
    import torch
    f = {"csr": asm.lib.fem_alls_consolidate, "bsr": asm.lib.fem_alls_consolidate_bsr,
         "upper": asm.lib.fem_alls_consolidate_upper}[form.split("_")[0]]
    off = 1 if form == "csr_unaligned" else 0
    ci = torch.empty(nnz + 65, dtype=torch.int32, device="cuda")
    v = torch.empty(nnz + 65, dtype=torch.float64, device="cuda")
    rp = torch.empty(asm.n_rows + 1, dtype=torch.int32, device="cuda")
    assert f(C.byref(asm.cm), C.byref(asm.opts), asm.ws_ptr, asm.ws_bytes, rp.data_ptr(), ci[off:].data_ptr(),
             v[off:].data_ptr(), nnz // asm.mesh.dpn ** 2 if form == "bsr" else nnz, asm._stream()) == 0
    return asm.read_info()[0]


def _fan_mesh():
    from test_gpu_rows2d import _fan
    return _fan(40, True)


@pytest.mark.parametrize("kind", ["q4", "t3", "t3_fan", "hex20", "hex20_ordered"])
@pytest.mark.parametrize("form", ["csr", "csr_unaligned", "bsr", "upper"])
@pytest.mark.parametrize("fault", ["lost_column", "count_too_small", "count_too_large"])
def test_lists_that_do_not_have_their_counts_columns(fem, cuda_device, kind, form, fault):
    # one row loses a column, or is counted with one less or (2-D) one more than it has: FEM_ERR_INTERNAL
    import torch
    if fault == "count_too_large" and (kind.startswith("hex20") or form == "upper"):
        pytest.skip("Hex20 lists keep what an earlier assembly left behind a row; the upper counts are taken from the list")
    m = _fan_mesh() if kind == "t3_fan" else _mesh(kind)
    asm = fem.Assembler(m)
    asm.ws.zero_()
    rp = asm.assemble()[0]
    nnz = int(rp[-1])
    assert _consolidate(asm, form, nnz) == 0
    n = 0 if kind == "t3_fan" else m.num_nodes // 2
    counts = _row_counts(torch, asm, rp)
    if fault == "lost_column":
        slots = _slots(torch, asm)[n, 2:]
        slots[int(torch.nonzero(slots).flatten()[-1])] = 0
    else:
        counts[n] += -1 if fault == "count_too_small" else 1
    assert _consolidate(asm, form, nnz + 64) == fem.FEM_ERR_INTERNAL
