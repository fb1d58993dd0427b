"""Completion stamps of fem_assemble_batched: each mesh's own, not its round's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_small_meshes_are_done_before_the_large_one_of_their_round(fem, cuda_device):
    # one round of four slots; the 2-D outputs are written before the Hex20 one, whose 24 M entries alone take 30 us at
    # any memory rate up to 10 TB/s
    import torch
    import meshgen as mg
    meshes = [mg.t3_grid(6, 5, seed=1), mg.hex20_grid(24, 24, 24, seed=1), mg.q4_grid(6, 5, seed=1), mg.mixed_grid(6, 5, seed=1)]
    b = fem.Batch(meshes, concurrency=4)
    b.sizes()
    # without an output a mesh is done once its size is known
    assert np.all(b.latencies_ms() > 0)
    for _ in range(3):
        b.run()
        torch.cuda.synchronize()
        assert all(s == 0 for s in b.statuses())
        lat = b.latencies_ms()
        assert np.all(lat > 0)
        assert np.all(np.delete(lat, 1) + 0.03 < lat[1]), lat
    # outputs too small for their meshes: done all the same, with the status
    for i in range(4):
        b.outs[i].capacity = 4
    b.stamps.zero_()
    b.run()
    torch.cuda.synchronize()
    assert b.statuses() == [1 << fem.FEM_ERR_CAPACITY] * 4
    assert np.all(b.latencies_ms() > 0)
