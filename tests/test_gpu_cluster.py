"""GPU: the LU and substitutions in one thread-block cluster (k_lu_cluster, the
graph form's default) against one kernel per elimination level
(gbpf_solver_set_lu_launch mode 1), over its schedules: the whole factor in one
CTA (small grids), cluster levels with a segment (chains of copies), with a
dense tail just over its least order, of 78 and with 43 levels before it, and
without either."""
import numpy as np
import pytest

from conftest import ieee_cases, ieee_path

pytestmark = pytest.mark.gpu


def grid_of(gb, name):
    if name.startswith("gen"):
        return gb.generate(4, 11, nbus=int(name[3:]))
    if name.startswith("ieee"):
        return gb.read_grid(ieee_path(next(c for c in ieee_cases() if c["cdf"] == name + ".cdf")))
    import bench

    return gb.read_grid(bench.grid_file(name))


# Two factorisations of one Jacobian differ by rounding only, and Newton ends on the same solution: in FP64 the last
# step's rounding is eps kappa |dx| with kappa <= 1e5 and |dx| <= 1e-2, below 1e-12 with room for the tiled grids'
# larger angles: 1e-11.  In FP32 the last step before max|g| <= 1e-10 is at most about 1e-5 and its relative error
# eps32 kappa <= 6e-3: 1e-7.
@pytest.mark.parametrize("precision,tol,atol", [("PREC_FP64", 1e-8, 1e-11), ("PREC_FP32_IR", 1e-10, 1e-7)])
@pytest.mark.parametrize("name", ["c4_14.cdf.gz", "gen15", "gen61", "c4_118.cdf.gz", "gen171", "c4_236.cdf.gz",
                                  "c4_472.cdf.gz", "ieee118x8", "c5_base.cdf.gz", "ieee118x64",
                                  "c3_base.cdfx.gz"])
def test_cluster_lu_matches_level_launches(gb, name, precision, tol, atol):
    grid = grid_of(gb, name)
    out = []
    for mode in (0, 1):
        s = gb.Solver(grid, tolerancia=tol, no_max_iter=100, lim_inj_reat=0, metodo=0, precision=getattr(gb, precision))
        s.set_form(gb.FORM_GRAPH)
        s.set_lu_launch(mode)
        out.append((s.info()["kernels_per_iteration"], s.solve(), s.solve()))
        s.close()
    (k0, a, a2), (k1, b, _) = out
    assert k0 < 12 < k1
    assert a["converged"] and b["converged"] and a["iterations"] == b["iterations"]
    for k in ("V", "theta"):
        np.testing.assert_allclose(a[k], b[k], rtol=0, atol=atol, err_msg=k)
        np.testing.assert_array_equal(a[k], a2[k])  # the same bits again


def test_cluster_lu_newton_step_and_singular(gb):
    """gbpf_newton_step through the cluster solves J dx = g (residual against the Jacobian the library returns), and an
    isolated bus (a zero pivot block) ends the solve with GBPF_E_SINGULAR."""
    grid = grid_of(gb, "c4_236.cdf.gz")
    s = gb.Solver(grid, tolerancia=1e-8, no_max_iter=100, metodo=0)
    b = grid.buses()
    V, th = b["V0"], b["theta0"] + 0.01 * np.sin(np.arange(grid.nB))
    row, col, val = s.eval_jacobian(V, th)
    n = int(row.max()) + 1
    g = np.cos(np.arange(n))
    dx = s.newton_step(V, th, g)
    J = np.zeros((n, n))
    J[row, col] = val
    assert np.max(np.abs(J @ dx - g)) <= 1e-13 * np.abs(J).sum(1).max() * np.abs(dx).max()
    iso = gb.create_grid(bus_type=[3, 0, 0, 0, 0], V0=[1.0] * 5, theta0=[0.0] * 5, from_bus=[1, 2, 3], to_bus=[2, 3, 4],
                         r=[0.01] * 3, x=[0.1] * 3, Pload=[0, 0.1, 0.1, 0.1, 0.1])
    s = gb.Solver(iso, tolerancia=1e-8, no_max_iter=10, metodo=0)
    s.set_form(gb.FORM_GRAPH)
    assert s.solve(full=False)["status"] == gb.E_SINGULAR


@pytest.mark.parametrize("name", ["ieee118x4", "ieee118x16"])
def test_persistent_form_on_request(gb, name):
    """Grids above the persistent form's default size still run it when asked, to the graph form's answer."""
    grid = grid_of(gb, name)
    s = gb.Solver(grid, tolerancia=1e-8, no_max_iter=100, metodo=0)
    assert s.form()["form"] == gb.FORM_GRAPH
    b = grid.buses()
    s.set_start(V0=b["V0"] * 1.001)  # before the form is built: its start is not the grid's own
    a = s.solve()
    s.set_form(gb.FORM_PERSISTENT)
    assert s.form()["form"] == gb.FORM_PERSISTENT
    p = s.solve()
    assert a["converged"] and a["iterations"] == p["iterations"]
    np.testing.assert_allclose(a["V"], p["V"], rtol=0, atol=1e-11)
    np.testing.assert_allclose(a["theta"], p["theta"], rtol=0, atol=1e-11)


@pytest.mark.parametrize("name,max_iter", [("c4_14.cdf.gz", 5), ("c4_14.cdf.gz", 300), ("c3_base.cdfx.gz", 3)])
def test_results_come_back_in_one_piece(gb, name, max_iter):
    """State and flows asked for array by array (any of them left out) are those of the whole result, below and above
    what one staged copy holds, and a history longer than what is read with the control record is all there: a solve
    that cannot reach its tolerance stops at no_max_iter with every iteration's mismatch."""
    import ctypes

    grid = grid_of(gb, name)
    s = gb.Solver(grid, tolerancia=1e-30, no_max_iter=max_iter, lim_inj_reat=0, metodo=0)
    r = s.solve()
    h = s.history()
    assert len(h) == r["iterations"] + 1 == max_iter + 1 and (h[:2] > 0).all()
    short = gb.Solver(grid, tolerancia=1e-30, no_max_iter=2, lim_inj_reat=0, metodo=0)
    np.testing.assert_array_equal(short.solve()["hist"], h[:3])
    for call, keys, n in (("gbpf_solver_state", ("V", "theta", "Pcalc", "Qcalc"), grid.nB),
                          ("gbpf_solver_flows", ("Pdp", "Ppd", "Qdp", "Qpd"), grid.nL)):
        for mask in range(16):
            a = [np.full(n, np.nan) for _ in range(4)]
            ptr = [x.ctypes.data_as(ctypes.c_void_p) if mask >> i & 1 else None for i, x in enumerate(a)]
            assert getattr(gb.lib(), call)(s.h, *ptr) == 0
            for i, k in enumerate(keys):
                np.testing.assert_array_equal(a[i], r[k] if mask >> i & 1 else np.full(n, np.nan), err_msg=k)


@pytest.mark.parametrize("precision", ["PREC_FP64", "PREC_FP32_IR"])
def test_profile_counts_the_substitutions_where_they_run(gb, precision):
    """The backward substitution is a phase of its own only where it is launched by itself: in the forms that take it
    with the factorisation its time and bytes are zero and its bytes are the factorisation's."""
    s = gb.Solver(grid_of(gb, "c5_base.cdf.gz"), tolerancia=1e-8, no_max_iter=100, metodo=0, precision=getattr(gb, precision))
    s.set_form(gb.FORM_GRAPH)
    s.solve(full=False)
    p = {}
    for mode in (0, 1, 2):
        s.set_lu_launch(mode)
        p[mode] = s.profile(3)
    assert p[1]["backward"]["ms"] > 0 and p[1]["backward"]["bytes"] > 0
    for mode in (0, 2):
        assert p[mode]["backward"] == dict(ms=0.0, bytes=0)
        assert p[mode]["factor_forward"]["ms"] > 0
        assert p[mode]["factor_forward"]["bytes"] == p[1]["factor_forward"]["bytes"] + p[1]["backward"]["bytes"]


# Backward error of a Newton step, |J dx - g| / (max row sum of |J| times |dx|): 1e-13 in FP64 as in the test of the
# 236-bus grid above, and 2^29 times that in FP32.
@pytest.mark.parametrize("precision,tol", [("PREC_FP64", 1e-13), ("PREC_FP32_IR", 1e-13 * 2 ** 29)])
@pytest.mark.parametrize("name", ["gen944", "tiles256"])
def test_cluster_lu_with_its_schedule_in_global_memory(gb, name, precision, tol):
    """Schedules that no CTA's shared memory holds: a filled 944-bus grid (lists of one int a pair) and a chain of 256
    copies of 118 buses, whose 80,375 factor blocks a triangle need lists of two ints a pair.  (That chain's Newton
    diverges from the flat start, on the CPU as well, so it is one Newton step that is held against the Jacobian.)"""
    sparse = pytest.importorskip("scipy.sparse")
    grid = gb.generate(3, 1, tiles=256) if name == "tiles256" else grid_of(gb, name)
    b = grid.buses()
    V, th = b["V0"], b["theta0"] + 0.01 * np.sin(np.arange(grid.nB))
    for mode in (0, 1):
        s = gb.Solver(grid, tolerancia=1e-8, no_max_iter=100, lim_inj_reat=0, metodo=0, precision=getattr(gb, precision))
        s.set_lu_launch(mode)
        info = s.info()
        assert info["factor_blocks"] > (65536 if name == "tiles256" else 16000)
        assert (info["kernels_per_iteration"] < 12) == (mode == 0)
        row, col, val = s.eval_jacobian(V, th)
        n = int(row.max()) + 1
        J = sparse.csr_matrix((val, (row, col)), shape=(n, n))
        g = np.cos(np.arange(n))
        dx = s.newton_step(V, th, g)
        assert np.isfinite(dx).all()
        assert np.abs(J @ dx - g).max() <= tol * abs(J).sum(axis=1).max() * np.abs(dx).max(), mode
        s.close()
