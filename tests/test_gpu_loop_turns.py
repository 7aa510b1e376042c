"""GPU: the graph loop's turns of several iterations, with the bank solves, the coarse
restriction and the stop test in one launch.  The host loop runs the same phases one iteration
at a time (and, with residual replacement, finishes the stop test in phase B): same sums in the
same order, so both loops must give the same bits for any iteration count (a turn's middle and
end), replacement interval (turns of 8, 4, 2 and 1 iterations) and level count (2 to 6 levels), as must
the separate launches of restriction, bank solves and stop test that the fused one replaces."""
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


@pytest.mark.parametrize("precond", ["mas", "diag"])
@pytest.mark.parametrize("precision,refine,turn", [("fp64", 32, 8), ("fp32", 32, 8), ("fp32", 12, 4), ("fp32", 3, 1)])
def test_reported_launches_count_whole_turns(dev, precond, precision, refine, turn):
    """kernel_launches of the graph loop: the kernels of every started turn, also past the stop,
    and two (one without MAS) per replacement; in FP64 a full turn is eight iterations of the host loop."""
    import torch
    from stgipc import PCGSolverConfig, Solver, scenes
    s = scenes.make_cube_drop(n=6, seed=4106)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    rows, cols, blocks, b = t(s.rows), t(s.cols), t(s.blocks.reshape(-1)), t(s.b)
    x = torch.zeros_like(b)

    def launches(iters, loop):
        v = Solver(PCGSolverConfig(precision=precision, stop_rule="relative_residual", global_tol_rate=1e-12, loop=loop,
                                   max_iter_ratio=(iters + 1.5) / s.n, refine_interval=refine, preconditioner=precond))
        if precond == "mas":
            v.mas_init(s.num_verts, s.neighbor_start, s.neighbor_num, s.neighbor_list, *s.slot_maps(16))
        v.solve_linear_system(rows, cols, blocks, b, x)  # loads modules, sizes buffers
        st = v.solve_linear_system(rows, cols, blocks, b, x)
        v.close()
        assert st["iterations"] == iters + 1  # the limit: `iters` ran
        return st["kernel_launches"] - st["replacements"] * (2 if precond == "mas" else 1)

    one = launches(1, "graph")
    assert launches(turn, "graph") == one
    per_turn = launches(turn + 1, "graph") - one
    assert per_turn > 0
    assert launches(2 * turn, "graph") == one + per_turn
    assert launches(2 * turn + 1, "graph") == one + 2 * per_turn
    if precision == "fp64":
        h1 = launches(1, "host")
        assert launches(9, "host") - h1 == per_turn
        assert launches(8, "host") == one


@pytest.mark.parametrize("n,bank,levels", [(6, 16, 4), (16, 16, 5), (40, 16, 6), (6, 32, 3), (16, 32, 4), (40, 32, 5)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_separate_launches_match_the_fused_one(dev, n, bank, levels, precision):
    """Recording samples for the learned correction takes the separate launches (restriction of
    level 2, of the levels above, bank solves, stop test in phase B), which very large systems and
    many scenes take too: the same bits as the fused launch, in both loops, for up to six levels
    of 16-vertex banks and five of 32-vertex ones."""
    import torch
    from stgipc import PCGSolverConfig, Solver, fem, scenes
    st = scenes.make_heterogeneous_cube(n=n, seed=4500 + n, state_only=True)
    V = st["pos"].shape[0]
    nb = scenes.vert_neighbors(V, st["tets"])
    maps = scenes.mas_partition_morton(V, bank)
    rows, cols, blocks, b = fem.newton_system(st["pos_rest"], st["pos"], st["vel"], st["tets"], st["E"], st["nu"], st["rho"],
                                              st["dt"], st["barriers"], device=dev)
    samples = torch.zeros(2, 4 * V, dtype=torch.float32, device=dev)
    for iters in (2, 17):
        got = []
        for loop, record in (("graph", False), ("host", False), ("graph", True), ("host", True)):
            v = Solver(PCGSolverConfig(precision=precision, stop_rule="relative_residual", global_tol_rate=1e-12, loop=loop,
                                       max_iter_ratio=(iters + 0.5) / (3 * V), bank_size=bank))
            v.mas_init(V, *nb, *maps)
            if record:
                v.net_configure(1)
                v.net_record(samples[0], samples[1], 1, 1000)
            x = torch.zeros_like(b)
            stats = v.solve_linear_system(rows, cols, blocks.reshape(-1), b, x)
            assert v.mas_info()[0] == levels
            assert (v.net_recorded() == 1) == record
            got.append((stats["iterations"], stats["rz_final"], stats["rel_residual_recursive"], x))
            v.close()
        for g in got[1:]:
            assert g[:3] == got[0][:3]
            assert torch.equal(g[3], got[0][3])
