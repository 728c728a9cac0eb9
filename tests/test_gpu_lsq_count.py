"""CSU_DUMP_LSQ_X87 counts (cell, variable) slots that the FP64 least squares leaves to the integer x87 model: once per
slot whatever the number of its components, and none where CSU_LSQ=x87 runs that model for everything."""
import pytest

pytestmark = pytest.mark.gpu


def _engine(monkeypatch, mode):
    import csu_b200
    from csu_b200 import meshgen
    if mode:
        monkeypatch.setenv("CSU_LSQ", mode)
    else:
        monkeypatch.delenv("CSU_LSQ", raising=False)
    su2, inp = meshgen.ramp(ni=24, nj=12)
    case = csu_b200.Case.from_text(inp, su2)
    U = case.initial_state()
    # a cell with three interior faces, its neighbours' too: one pressure beyond the range the FP64 path decides in
    # (2^961) puts the variable p of the cell and of its three neighbours on the integer model, no other variable
    nint = case.cell_nint
    nei = [case.con[case.con[:, 0] == c, 1].tolist() + case.con[case.con[:, 1] == c, 0].tolist()
           for c in range(case.n_cells)]
    c0 = next(c for c in range(case.n_cells) if nint[c] == 3 and all(nint[n] == 3 for n in nei[c]))
    U[3, c0] = 1e300
    return csu_b200.Engine(case, state=U)


def test_one_count_per_variable(native, monkeypatch):
    eng = _engine(monkeypatch, None)
    eng.residual()
    assert eng.dump("LSQ_X87")[0] == 4
    eng.residual()
    assert eng.dump("LSQ_X87")[0] == 8
    eng.close()


def test_x87_mode_counts_nothing(native, monkeypatch):
    eng = _engine(monkeypatch, "x87")
    eng.residual()
    assert eng.dump("LSQ_X87")[0] == 0
    eng.close()


def test_x87_mode_costs_what_it_has_to(native, monkeypatch):
    """The integer model is a few hundred instructions a component more, no more than that: an RK5 iteration with it
    takes under three times one without (60,000 cells; both sides the best of five)."""
    import time
    import csu_b200
    from csu_b200 import meshgen
    su2, inp = meshgen.bump(ncells=60000, mach=0.5, order=2, scheme="RK", cfl=0.5, flux="AUSM")
    case = csu_b200.Case.from_text(inp, su2)
    best = {}
    for mode in (None, "x87"):
        if mode:
            monkeypatch.setenv("CSU_LSQ", mode)
        else:
            monkeypatch.delenv("CSU_LSQ", raising=False)
        eng = csu_b200.Engine(case)
        eng.iterate(8)
        t = []
        for _ in range(5):
            a = time.perf_counter()
            eng.iterate(8)
            t.append(time.perf_counter() - a)
        best[mode] = min(t)
        eng.close()
    assert best["x87"] < 3.0 * best[None], best
