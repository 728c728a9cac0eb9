"""The WIDE build of the DPLUR sweeps (meshes of more than one wave of the other) against the PLAIN one: two solves of
half a WIDE mesh in one pack, whose cells add up, equal each solve alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("viscous", [None, "laminar"])
@pytest.mark.parametrize("fp32", [0, 1])
def test_wide_equals_plain(native, monkeypatch, viscous, fp32):
    import csu_b200
    import torch
    from csu_b200 import meshgen
    monkeypatch.setenv("CSU_AUTOTUNE", "0")
    # a third of a multiprocessor's PLAIN cells more than half: 427 and 854 cells a multiprocessor
    n = torch.cuda.get_device_properties(0).multi_processor_count * 427
    su2, inp = meshgen.bump(ncells=n, mach=0.5, viscous=viscous, re=1e4 if viscous else None, order=1, n_linear=5,
                            cfl=2.0, flux="AUSM")
    case = csu_b200.Case.from_text(inp + "implicitFP32, %d\n" % fp32, su2)
    U = case.initial_state()
    rng = np.random.default_rng(3)
    states = [U * (1 + 0.01 * rng.uniform(-1, 1, U.shape)) for _ in range(2)]
    alone = []
    for s in states:
        eng = csu_b200.Engine(case, state=s)
        eng.iterate(4)
        alone.append(eng.get_state())
        eng.close()
    pack = csu_b200.Pack([csu_b200.Prep(case, state=s) for s in states])
    pack.iterate(4)
    for k in range(2):
        assert np.array_equal(pack.get_state(k), alone[k])
    pack.close()
