"""CSU_DUMP_SST_JAC outside SST is refused, also where an SA context keeps its own implicit source in the same array (one
row, not the view's six)."""
import pytest

import casekit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("implicit_source", ["0", "1"])
def test_refused_with_sa(native, implicit_source):
    import csu_b200
    wd = casekit.materialize("caseBL_turb", {"restart": "0", "order": "1", "timeScheme": "DPLUR", "Nlinear": "4",
                                             "CFL": "2.0", "saImplicitSource": implicit_source})
    eng = csu_b200.Engine(csu_b200.Case.load(wd))
    eng.iterate(2)
    with pytest.raises(csu_b200.CsuError) as e:
        eng.dump("SST_JAC")
    assert "no SST source Jacobians" in str(e.value)
    eng.close()
