"""Builds of one kernel chosen by mesh size (csu_b200/csrc/cuda/launch_rules.h) give the same bits: several solves in one
pack, whose cells add up to another build's sizes, equal each solve alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(per_sm, solves, viscous, **solver):
    """`solves` disturbed states on a mesh of per_sm cells a multiprocessor, alone and in one pack, four iterations."""
    import csu_b200
    import torch
    from csu_b200 import meshgen
    fp32 = solver.pop("fp32", 0)
    n = torch.cuda.get_device_properties(0).multi_processor_count * per_sm
    su2, inp = meshgen.bump(ncells=n, mach=0.5, viscous=viscous, re={None: None, "laminar": 1e4}.get(viscous, 2e6),
                            flux="AUSM", **solver)
    case = csu_b200.Case.from_text(inp + "implicitFP32, %d\n" % fp32, su2)
    U = case.initial_state()
    rng = np.random.default_rng(3)
    states = [U * (1 + 0.01 * rng.uniform(-1, 1, U.shape)) for _ in range(solves)]
    alone = []
    for s in states:
        eng = csu_b200.Engine(case, state=s)
        eng.iterate(4)
        alone.append(eng.get_state())
        eng.close()
    pack = csu_b200.Pack([csu_b200.Prep(case, state=s) for s in states])
    pack.iterate(4)
    for k in range(solves):
        assert np.array_equal(pack.get_state(k), alone[k])
    pack.close()


@pytest.mark.parametrize("viscous", [None, "laminar"])
@pytest.mark.parametrize("fp32", [0, 1])
def test_wide_equals_plain(native, monkeypatch, viscous, fp32):
    """Sweeps: 427 cells a multiprocessor PLAIN, 854 WIDE (more than the 640 of one PLAIN wave)."""
    monkeypatch.setenv("CSU_AUTOTUNE", "0")
    _compare(427, 2, viscous, order=1, n_linear=5, cfl=2.0, fp32=fp32)


@pytest.mark.parametrize("viscous", [None, "laminar", "sa"])
@pytest.mark.parametrize("fp32", [0, 1])
def test_early_equals_plain(native, monkeypatch, viscous, fp32):
    """Sweeps: 128 cells a multiprocessor EARLY, 384 PLAIN."""
    monkeypatch.setenv("CSU_AUTOTUNE", "0")
    _compare(128, 3, viscous, order=1, n_linear=5, cfl=2.0, fp32=fp32)


@pytest.mark.parametrize("viscous", [None, "laminar", "sa", "sst"])
def test_small_gradients_equal_the_others(native, monkeypatch, viscous):
    """Gradients: half a block of 32 cells a multiprocessor SMALL, four blocks not."""
    monkeypatch.setenv("CSU_AUTOTUNE", "0")
    _compare(16, 8, viscous, order=2, scheme="RK", cfl=0.5)
