"""GPU: the graph loop's turns of several iterations, with the bank solves, the coarse
restriction and the stop test in one launch.  The host loop runs the same phases one iteration
at a time (and, with residual replacement, finishes the stop test in phase B): same sums in the
same order, so both loops must give the same bits for any iteration count (a turn's middle and
end), replacement interval (turns of 8, 4, 2 and 1 iterations) and level count (2 to 5 levels)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(dev, s, loop, precision, refine, ratio, bank=16):
    import torch
    from stgipc import GlobalLinearSystem, PCGSolverConfig
    g = GlobalLinearSystem(s, PCGSolverConfig(precision=precision, stop_rule="relative_residual", global_tol_rate=1e-9,
                                              max_iter_ratio=ratio, refine_interval=refine, loop=loop, bank_size=bank),
                           device=dev)
    st = g.solve_linear_system()
    torch.cuda.synchronize()
    x = g.x.cpu().numpy()
    g.solver.close()
    return st, x


@pytest.mark.parametrize("n", [1, 3, 6, 16])
@pytest.mark.parametrize("bank", [16, 32])
@pytest.mark.parametrize("precision,refine", [("fp64", 32), ("fp32", 32), ("fp32", 12), ("fp32", 6), ("fp32", 3), ("fp32", 1)])
def test_turns_match_single_iterations(dev, n, bank, precision, refine):
    from oracle import oracle as orc
    from stgipc import scenes
    s = scenes.make_cube_drop(n=n, seed=4100 + n)
    dof = 3 * s.num_verts
    rows, cols, blocks = orc.convert(s.rows, s.cols, s.blocks)
    for iters in (2, 7, 8, 9, 17):
        ratio = (iters + 0.5) / dof
        sg, xg = _solve(dev, s, "graph", precision, refine, ratio, bank)
        sh, xh = _solve(dev, s, "host", precision, refine, ratio, bank)
        assert sg["iterations"] == sh["iterations"] and sg["status"] == sh["status"]
        assert sg["replacements"] == sh["replacements"]
        assert sg["rel_residual_recursive"] == sh["rel_residual_recursive"]
        np.testing.assert_array_equal(xg, xh)
    # to convergence: the residual of the oracle's product
    sg, xg = _solve(dev, s, "graph", "fp64", refine, 20.0, bank)
    assert sg["status"] == 0
    r = s.b - orc.spmv(rows, cols, blocks, xg)
    assert np.linalg.norm(r) <= 1.01e-9 * np.linalg.norm(s.b) + 1e-13 * np.linalg.norm(s.b) * dof


@pytest.mark.parametrize("precision,refine", [("fp64", 32), ("fp32", 32), ("fp32", 5)])
@pytest.mark.parametrize("count", [1, 17, 40])
def test_scene_turns_match_single_iterations(dev, count, precision, refine):
    """Scenes with their own stop tests (one CTA each beside the bank solves; more than one
    cluster of them at 17 and 40): graph and host loop end every scene at the same iteration
    with the same bits, at convergence and when the iteration limit ends the loop first."""
    import torch
    from stgipc import PCGSolverConfig, scenes
    from stgipc.batch import ConcatenatedBatch
    sysl = scenes.make_batched_cubes(count=count, seed=4300, n_lo=3, n_hi=7)
    dof = sum(s.n for s in sysl)
    for ratio in (0.3, 9.5 / dof):
        got = []
        for loop in ("graph", "host"):
            cb = ConcatenatedBatch(sysl, PCGSolverConfig(precision=precision, refine_interval=refine, loop=loop,
                                                         max_iter_ratio=ratio), device=dev, spmv_tiles=-1)
            st = cb.solve()
            torch.cuda.synchronize()
            it, rel = cb.scene_stats()
            got.append((st["status"], st["iterations"], it.tolist(), rel.tolist(), cb.x.cpu().numpy()))
            cb.close()
        assert got[0][:4] == got[1][:4]
        np.testing.assert_array_equal(got[0][4], got[1][4])
        if ratio == 0.3:
            assert got[0][0] == 0 and max(got[0][3]) <= 1e-4
