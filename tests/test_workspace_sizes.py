"""Workspace sizes that callers saved stay valid: fem_alls_workspace_size answers
what it always has, the sum of the regions below (a restatement of the library's
original layout), for every kind and option, but for Hex20 meshes with more than
half as many elements as nodes; fem_batched_workspace_size no more than it has
(its first batches also had a control block)."""
import ctypes as C

import pytest

up = lambda v: -(-v // 256) * 256  # noqa: E731
HEX20 = 2


def _original(kind, N, E, first=0, more=0, pool=0.0):
    dpn = 3 if kind == HEX20 else 2
    s1, s2 = (first or 94, more or 30) if dpn == 3 else (14, 14)
    x = (pool or (0.5 if dpn == 3 else 0.125)) * N
    cap2 = int(x) + (int(x) < x) + 64
    slots = N * s1 + cap2 * s2
    bits = 1
    while bits < 5 and 8 ** bits * 4 < E:
        bits += 1
    buckets = 8 ** bits if dpn == 3 else 2 * ((N >> 8) + 1)
    total = 256 + up(N * (s1 + 2) * 4) + up(cap2 * (s2 + 2) * 4) + up(slots * dpn * dpn * 8) + 2 * up(N * 4)
    total += up(-(-N // 4096) * 8) + up(E * 4) + 256 + up(buckets * 4) + 256
    if kind == HEX20:
        total += 2 * up((N + 1) * 4) + up(E * 80) + up(-(-min(E, 32768) // 8) * 20880)
    return total


def _mesh(fem, kind, N, E):
    stride = {0: 4, 1: 3, 2: 20, 3: 4}[kind]
    return fem.FemMesh(kind, N, E, stride, *([256] * 5), None, None, 1.0, 0.3, 1.0)


def _size(fem, m, o=None):
    n = C.c_size_t()
    assert fem.load().fem_alls_workspace_size(C.byref(m), C.byref(o) if o else None, C.byref(n)) == 0
    return n.value


def _hex_grid(n):
    return (n + 1) ** 3 + 3 * n * (n + 1) ** 2, n ** 3


@pytest.mark.parametrize("n", [1, 2, 3, 9, 14, 15, 20, 32, 33, 40, 47, 48, 64, 65, 80, 100])
def test_hex20_grids(fem, n):
    N, E = _hex_grid(n)
    assert _size(fem, _mesh(fem, HEX20, N, E)) == _original(HEX20, N, E)
    for first, more, pool in ((62, 30, 1.0), (46, 30, 1.0), (94, 10, 0.25)):
        o = fem.opts(first_slots=first, chunk_slots=more, pool_factor=pool)
        assert _size(fem, _mesh(fem, HEX20, N, E), o) == _original(HEX20, N, E, first, more, pool)


@pytest.mark.parametrize("kind", [0, 1, 3])
@pytest.mark.parametrize("N,E", [(1, 0), (4, 1), (1111, 1000), (4096, 8000), (4097, 8000), (700000, 1400000), (2250000, 3400000)])
def test_2d(fem, kind, N, E):
    assert _size(fem, _mesh(fem, kind, N, E)) == _original(kind, N, E)
    assert _size(fem, _mesh(fem, kind, N, E), fem.opts(pool_factor=1.0)) == _original(kind, N, E, pool=1.0)


@pytest.mark.parametrize("N,E", [(20, 0), (20, 1), (1000, 500), (100000, 50000), (300000, 140000), (1000000, 10)])
def test_hex20_up_to_half_as_many_elements_as_nodes(fem, N, E):
    assert _size(fem, _mesh(fem, HEX20, N, E)) == _original(HEX20, N, E)


@pytest.mark.parametrize("N,E", [(81, 320), (1000, 2000), (100000, 100000)])
def test_hex20_with_more_elements_has_room_for_them(fem, N, E):
    # packed Ke and rank map of every element, 15,120 + 800 bytes
    assert _original(HEX20, N, E) <= _size(fem, _mesh(fem, HEX20, N, E)) <= _original(HEX20, N, E) + 15920 * E + N + 1024


@pytest.mark.parametrize("grids", [(33, 20), (48, 33, 9), (50, 50)])
def test_batches(fem, grids):
    # one slot per mesh: a control unit, and per Hex20 slot the records of 4,096 elements
    ms = [_mesh(fem, HEX20, *_hex_grid(n)) for n in grids]
    b = C.c_size_t()
    assert fem.load().fem_batched_workspace_size((fem.FemMesh * len(ms))(*ms), len(ms), None, len(ms), C.byref(b)) == 0
    want = sum(_original(HEX20, *_hex_grid(n)) + up(-(-min(n ** 3, 4096) // 8) * 20880) for n in grids)
    assert b.value == 256 + want
