"""The BLOCKS view unpacks the stored entries of the 32-cell tiles: FP32 blocks are the rounded FP64 ones entry by entry,
entries the operator never has and slots without a face are zero, on cell counts beside a tile's edge."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("viscous,nvar", [(None, 4), ("sa", 5), ("sst", 6)])
@pytest.mark.parametrize("cells", [250, 1000])
def test_blocks_view(native, viscous, nvar, cells):
    import csu_b200
    from csu_b200 import meshgen
    su2, inp = meshgen.bump(ncells=cells, mach=0.5, viscous=viscous, re=2e6 if viscous else None, order=1, n_linear=4,
                            cfl=1.0, flux="AUSM")
    views = []
    for fp32 in (0, 1):
        case = csu_b200.Case.from_text(inp + "implicitFP32, %d\n" % fp32, su2)
        assert case.n_cells % 32
        eng = csu_b200.Engine(case)
        eng.iterate(1)
        views.append(eng.dump("BLOCKS"))
        eng.close()
    f64, f32 = views
    assert np.array_equal(f64.astype(np.float32).astype(np.float64), f32)
    assert not f64[:, :, 0, 3:].any() and np.isfinite(f64).all()
    for r in range(4, nvar):
        assert not f64[:, :, r, [k for k in range(3, nvar) if k != r]].any()
    for j in range(4):
        absent = case.cell_nint <= j
        assert not f64[absent, j].any() and f64[~absent, j, 0, 0].all()
