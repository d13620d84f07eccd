"""GPU: the persistent form asked for (gbpf_solver_set_form) on every golden grid whose state fits one block, the ones
above its default size among them, and every LU plan of it (gbpf_solver_set_plan).  Only a grid that the library itself
refuses (GBPF_E_UNSUPPORTED) is passed over, and only where the factor in FP64 really is larger than a block's shared
memory.  Tolerances are those of the parity tests: identical iterations and switch events, |V| and theta within 1e-9,
the mismatch of each iteration within 1e-6 relative."""
import numpy as np
import pytest

from conftest import case_path, committed_cases, ieee_cases, load_golden
from test_gpu_parity import check_solution, solver

pytestmark = pytest.mark.gpu


def persistent(gb, case):
    grid, s = solver(gb, case_path(case), tolerancia=case["tol"], no_max_iter=case["max_iter"],
                     lim_inj_reat=case["lim"])
    try:
        s.set_form(gb.FORM_PERSISTENT)
    except gb.GbpfError as e:
        assert e.status == gb.E_UNSUPPORTED and grid.nB > 2000, (e, grid.nB)
        pytest.skip("the grid's state does not fit one block's shared memory")
    form = s.form()
    assert form["form"] == gb.FORM_PERSISTENT and form["launches"] <= 2
    return s


@pytest.mark.parametrize("case", committed_cases() + ieee_cases(), ids=lambda c: c["golden"])
def test_persistent_form_matches_reference_golden(gb, case):
    s = persistent(gb, case)
    gold = load_golden(case["golden"])
    res = s.solve()
    check_solution(res, gold)
    h = np.array(gold["hist"])[:-1] if gold["converged"] else np.array(gold["hist"])[:10]
    np.testing.assert_allclose(res["hist"][:len(h)], h, rtol=1e-6, atol=1e-12)


@pytest.mark.parametrize("plan", [(1, 0, 1), (1, 0, 0), (1, 1, 1), (0, 0, 1), (0, 1, 0)],
                         ids=lambda p: f"lu1={p[0]},narrow={p[1]},quad={p[2]}")
@pytest.mark.parametrize("case", [c for c in ieee_cases(max_buses=1888)
                                  if c["golden"] in ("ieee_ieee118x4_lim0.json", "ieee_ieee118x16_lim0.json.gz")],
                         ids=lambda c: c["golden"])
def test_persistent_plans_on_request_match_reference_golden(gb, case, plan):
    s = persistent(gb, case)
    want = dict(lu1=plan[0], narrow=plan[1], quad=plan[2])
    assert s.set_plan(*plan) == want
    assert s.set_plan() == want
    check_solution(s.solve(), load_golden(case["golden"]))
