"""fem_autotune varies only options that the mesh's kind uses, and keeps the others."""
import pytest

pytestmark = pytest.mark.gpu


def test_hex20_keeps_the_grid_option(fem, cuda_device):
    import meshgen as mg
    asm = fem.Assembler(mg.hex20_grid(4, seed=1), fem.opts(ctas_per_sm=7))
    best, ms = asm.autotune(repeats=1)
    assert best.ctas_per_sm == 7 and best.first_slots in (94, 62, 46) and best.chunk_slots == 30 and ms > 0.0


@pytest.mark.parametrize("kind", ["q4_grid", "t3_grid", "mixed_grid"])
def test_2d_keeps_the_list_options(fem, cuda_device, kind):
    import meshgen as mg
    asm = fem.Assembler(getattr(mg, kind)(9, 8, seed=1), fem.opts(pool_factor=0.75, precision=fem.FEM_PREC_FP32))
    best, ms = asm.autotune(repeats=1)
    assert best.ctas_per_sm in (0, 1, 2, 3) and best.first_slots == best.chunk_slots == 0
    assert best.pool_factor == 0.75 and best.precision == fem.FEM_PREC_FP32 and ms > 0.0
