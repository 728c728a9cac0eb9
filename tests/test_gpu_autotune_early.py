"""The autotuner on meshes whose DPLUR sweeps are the EARLY build: it reports the 64-cell blocks they run in."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("per_sm", [112, 150, 190])
def test_reported_shape_is_the_one_that_runs(native, fp32, per_sm):
    import csu_b200
    import torch
    from csu_b200 import meshgen
    n = torch.cuda.get_device_properties(0).multi_processor_count * per_sm
    nj = int(round((n / 4.0) ** 0.5))
    su2, inp = meshgen.ramp(ni=n // (2 * nj), nj=nj, n_linear=4, cfl=5.0)
    eng = csu_b200.Engine(csu_b200.Case.from_text(inp + "implicitFP32, %d\n" % fp32, su2))
    for _ in range(3):
        assert eng.autotune()[1] == 64
    eng.close()
