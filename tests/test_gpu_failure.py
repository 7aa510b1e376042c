"""GPU: the bounded device waits give up instead of hanging, report STG_ERR_TIMEOUT, and
leave the context usable (no fault, trap or endless loop is involved: the waited-on
mbarrier is simply never completed)."""
import ctypes as C

import numpy as np
import pytest

from conftest import cube_system

pytestmark = pytest.mark.gpu


def test_bounded_wait_gives_up_and_context_stays_usable(dev):
    import torch
    from stgipc import GlobalLinearSystem, PCGSolverConfig, _lib
    L = _lib.lib()
    status, seconds = C.c_int(-1), C.c_double(-1.0)
    assert L.stg_selftest_wait_timeout(C.byref(status), C.byref(seconds)) == _lib.STG_OK
    assert status.value == _lib.STG_ERR_TIMEOUT
    # every bounded wait gives up after 1 s of the device's global timer
    assert 0.9 < seconds.value < 3.0, seconds.value
    # the device still works: a normal solve afterwards
    gls = GlobalLinearSystem(cube_system(8), PCGSolverConfig(), device=dev)
    st = gls.solve_linear_system()
    assert st["status"] == _lib.STG_OK and np.isfinite(gls.x.cpu().numpy()).all()
    torch.cuda.synchronize()


@pytest.mark.parametrize("where,prec,loop", [("b", "fp64", "graph"), ("b", "fp32", "graph"),
                                             ("block", "fp32", "host"), ("block", "fp64", "graph")])
def test_nan_input_reports_breakdown(dev, where, prec, loop):
    """A NaN in the right-hand side or in one Hessian block (a corrupted input, injected on
    the host) ends the solve at once with STG_BREAKDOWN instead of iterating on NaNs; the
    handle then solves a clean system normally."""
    import numpy as np
    import torch
    from conftest import cube_system
    from stgipc import PCGSolverConfig, Solver, StgError, _lib
    s = cube_system(8)
    solver = Solver(PCGSolverConfig(precision=prec, loop=loop, stop_rule="relative_residual"))
    solver.mas_init(s.num_verts, s.neighbor_start, s.neighbor_num, s.neighbor_list, *s.slot_maps(16))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    b = s.b.copy()
    blocks = s.blocks.copy()
    if where == "b":
        b[17] = np.nan
    else:
        blocks[len(blocks) // 2, 4] = np.nan
    x = t(np.zeros(s.n))
    with pytest.raises(StgError) as e:
        solver.solve_linear_system(t(s.rows), t(s.cols), t(blocks.reshape(-1)), t(b), x)
    assert e.value.status == _lib.STG_BREAKDOWN
    st = solver.solve_linear_system(t(s.rows), t(s.cols), t(s.blocks.reshape(-1)), t(s.b), x)
    assert st["status"] == 0 and st["rel_residual"] <= 1.2e-4


@pytest.mark.parametrize("site", [0, 1])
@pytest.mark.parametrize("loop,precision,refine,bank,precond", [
    ("graph", "fp64", 32, 16, "mas"), ("graph", "fp64", 32, 32, "mas"), ("graph", "fp64", 32, 16, "diag"),
    ("graph", "fp32", 32, 16, "mas"), ("graph", "fp32", 3, 16, "mas"), ("graph", "fp32", 32, 16, "diag"),
    ("host", "fp64", 32, 16, "mas")])
def test_wait_that_gives_up_ends_the_loop(dev, site, loop, precision, refine, bank, precond):
    """An iteration marked as if a bounded wait had given up in its SpMV phase or bank solves (a
    kernel records the error; nothing waits): the captured loop ends with that turn and the solve
    reports STG_ERR_TIMEOUT, also when the stop test had set the loop to go on.  The handle then
    solves as a fresh one does."""
    import torch
    from stgipc import PCGSolverConfig, Solver, StgError, _lib
    L = _lib.lib()
    s = cube_system(8)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    rows, cols, blocks, b = t(s.rows), t(s.cols), t(s.blocks.reshape(-1)), t(s.b)

    def make():
        v = Solver(PCGSolverConfig(precision=precision, loop=loop, stop_rule="relative_residual", global_tol_rate=1e-9,
                                   refine_interval=refine, bank_size=bank, preconditioner=precond))
        if precond == "mas":
            v.mas_init(s.num_verts, s.neighbor_start, s.neighbor_num, s.neighbor_list, *s.slot_maps(bank))
        return v

    fresh, solver = make(), make()
    want, x = torch.zeros_like(b), torch.zeros_like(b)
    st0 = fresh.solve_linear_system(rows, cols, blocks, b, want)
    assert st0["iterations"] > 10
    for iteration in (1, 2, 8, 9):
        assert L.stg_selftest_fail_iteration(solver.h, iteration, site) == _lib.STG_OK
        with pytest.raises(StgError) as e:
            solver.solve_linear_system(rows, cols, blocks, b, x)
        assert e.value.status == _lib.STG_ERR_TIMEOUT
    assert L.stg_selftest_fail_iteration(solver.h, 0, 0) == _lib.STG_OK
    st = solver.solve_linear_system(rows, cols, blocks, b, x)
    assert st["status"] == st0["status"] and st["iterations"] == st0["iterations"]
    assert torch.equal(x, want)
    fresh.close()
    solver.close()
