"""GPU: the Hessian producer (stg_fem_newton_system) against the CPU assembly of the
synthetic scenes (stgipc/scenes._assemble): same converted BCOO pattern, blocks and
gradient to FP64 rounding (summation order and eigen-solver differ), barriers active on
both planes, and the solve of the GPU-built system matching the CPU-built one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,seed", [(6, 2400), (10, 2401)])
def test_newton_system_matches_cpu_assembly(dev, n, seed):
    from oracle import oracle as orc
    from stgipc import fem, scenes
    st = scenes.make_heterogeneous_cube(n=n, seed=seed, state_only=True)
    cpu = scenes._assemble(**st)
    rows, cols, blocks, b = fem.newton_system(st["pos_rest"], st["pos"], st["vel"], st["tets"], st["E"], st["nu"],
                                              st["rho"], st["dt"], st["barriers"], device=dev)
    assert rows.numel() == 10 * st["tets"].shape[0] + cpu.num_verts
    rg, cg, bg = orc.convert(rows.cpu().numpy(), cols.cpu().numpy(), blocks.cpu().numpy())
    rc, cc, bc = orc.convert(cpu.rows, cpu.cols, cpu.blocks)
    np.testing.assert_array_equal(rg, rc)
    np.testing.assert_array_equal(cg, cc)
    scale = np.abs(bc).max()
    assert np.abs(bg - bc).max() <= 1e-10 * scale
    bb = b.cpu().numpy()
    assert np.abs(bb - cpu.b).max() <= 1e-10 * np.abs(cpu.b).max()
    # both barrier planes are active in this state
    y = st["pos"][:, 1]
    assert (y < st["barriers"][0][2]).any() and ((-y + st["barriers"][1][1]) < st["barriers"][1][2]).any()


def test_gpu_built_system_solves_like_cpu_built(dev):
    import torch
    from stgipc import PCGSolverConfig, Solver, fem, scenes
    st = scenes.make_heterogeneous_cube(n=12, seed=2402, state_only=True)
    cpu = scenes._assemble(**st)
    rows, cols, blocks, b = fem.newton_system(st["pos_rest"], st["pos"], st["vel"], st["tets"], st["E"], st["nu"],
                                              st["rho"], st["dt"], st["barriers"], device=dev)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    out = []
    for R, C, B, bb in ((rows, cols, blocks.reshape(-1), b), (t(cpu.rows), t(cpu.cols), t(cpu.blocks.reshape(-1)),
                                                               t(cpu.b))):
        s = Solver(PCGSolverConfig(precision="fp64", stop_rule="relative_residual", global_tol_rate=1e-6))
        s.mas_init(cpu.num_verts, cpu.neighbor_start, cpu.neighbor_num, cpu.neighbor_list, *cpu.slot_maps(16))
        x = torch.zeros_like(bb)
        stt = s.solve_linear_system(R, C, B, bb, x)
        out.append((stt["iterations"], x.cpu().numpy()))
    assert abs(out[0][0] - out[1][0]) <= 1
    assert np.linalg.norm(out[0][1] - out[1][1]) <= 1e-6 * np.linalg.norm(out[1][1])


@pytest.mark.parametrize("T", [1, 31, 33, 129, 300])
def test_closed_form_projection_on_hard_tets(dev, T):
    """The closed-form PSD projection against numpy's eigh, per tet: strongly compressed,
    inverted, flattened, collapsed and rank-one deformations, a negative modulus, warps that are
    not full, and one vertex shared by every tet (more incident tets than are sorted in registers).  Both projections are backward stable, so they agree to a few hundred eps of the
    unprojected Hessian's norm in x (kinetic scale max d^2): 1e-12."""
    from stgipc import fem, scenes
    rng = np.random.default_rng(77 + T)
    rest = rng.normal(size=(3 * T + 1, 3))
    tets = np.stack([np.zeros(T, np.int64), 3 * np.arange(T) + 1, 3 * np.arange(T) + 2, 3 * np.arange(T) + 3], 1)
    rest[0] = 0.0
    Dm = np.transpose(rest[tets[:, 1:]], (0, 2, 1))
    for t in range(T):  # well-shaped rest tets
        q, _ = np.linalg.qr(Dm[t])
        rest[tets[t, 1:]] = (q + 0.2 * rng.uniform(-1, 1, (3, 3))).T
    F = np.eye(3) + rng.normal(scale=0.6, size=(T, 3, 3))
    kind = np.arange(T) % 7
    F[kind == 1] *= 0.05
    F[kind == 2, :, 0] *= -1.0
    F[kind == 3, :, 2] = F[kind == 3, :, 1]
    F[kind == 4] = 0.0
    F[kind == 5, :, 1:] = 2.0 * F[kind == 5, :, :1]
    pos = rest.copy()
    for t in range(T):
        pos[tets[t, 1:]] = rest[tets[t, 1:]] @ F[t].T
    E = np.exp(rng.uniform(np.log(1e3), np.log(1e6), T))
    E[kind == 6] *= -1.0
    st = dict(pos_rest=rest, pos=pos, vel=np.zeros_like(pos), tets=tets, E=E, nu=0.45, rho=1000.0, dt=0.01, barriers=[])
    cpu = scenes._assemble(name="hard", **st)
    rows, cols, blocks, b = fem.newton_system(rest, pos, st["vel"], tets, E, 0.45, 1000.0, 0.01, device=dev)
    np.testing.assert_array_equal(rows.cpu().numpy(), cpu.rows)
    np.testing.assert_array_equal(cols.cpu().numpy(), cpu.cols)
    got = blocks.cpu().numpy()[:10 * T].reshape(T, 90)
    ref = cpu.blocks[:10 * T].reshape(T, 90)
    # scale: |H9| <= |mu| + |lam| |g|^2 + |lam (J - alpha)| |F|, times vol dt^2 |d|^2
    Dm = np.transpose(rest[tets[:, 1:]] - rest[tets[:, :1]], (0, 2, 1))
    Ff = np.transpose(pos[tets[:, 1:]] - pos[tets[:, :1]], (0, 2, 1)) @ np.linalg.inv(Dm)
    mu, lam = np.abs(E) / 2.9, np.abs(E) * 0.45 / (1.45 * 0.1)
    f = np.linalg.norm(Ff, axis=(1, 2))
    h = mu + lam * f ** 4 + lam * (f ** 3 + 2.0) * f
    d2 = (np.linalg.norm(np.linalg.inv(Dm), axis=(1, 2)) ** 2) * 4
    scale = np.abs(np.linalg.det(Dm)) / 6.0 * 1e-4 * d2 * h
    assert (np.abs(got - ref).max(axis=1) <= 1e-12 * scale).all()
    np.testing.assert_allclose(b.cpu().numpy(), cpu.b, atol=1e-12 * T * np.abs(cpu.b).max())


def _degenerate_gradients():
    """Deformation gradients of rank zero to two with the non-zero columns in every place, and
    with columns whose squares vanish in 64 bits."""
    a, b = np.array([0.6, 0.7, -0.5]), np.array([-0.3, 1.1, 0.4])
    out = [np.zeros((3, 3))]
    for c in range(3):
        for s in (1.0, 2.5):
            F = np.zeros((3, 3))
            F[:, c] = s * a
            out.append(F)                       # rank one, the other columns exactly zero
            for tiny in (1e-100, 1e-160, 1e-170):
                G = F.copy()
                G[:, (c + 1) % 3] = tiny * a    # parallel to the lone column
                out.append(G)
                G = G.copy()
                G[:, (c + 2) % 3] = 0.5 * tiny * b
                out.append(G)
        for tiny in (0.0, 1e-120, 1e-168):
            F = np.stack([a, b, a - 2.0 * b], 1)
            F[:, c] = tiny
            out.append(F)                       # rank two
    out += [np.diag([s, s, q]) for s in (1.0, 2.0) for q in (1e-150, 1e-172, 1e-200)]
    out += [q * np.eye(3) for q in (1e-60, 1e-150, 1e-200)]
    return np.stack(out)


def test_closed_form_projection_of_degenerate_gradients(dev):
    """Against numpy's eigh, as above, on unit rest tets (F is exact): 1e-12 of the unprojected
    Hessian's bound, and no NaN where eigh has none."""
    from stgipc import fem, scenes
    F = _degenerate_gradients()
    T = F.shape[0]
    rest = np.tile(np.concatenate([np.zeros((1, 3)), np.eye(3)]), (T, 1))
    tets = np.arange(4 * T).reshape(T, 4)
    pos = np.zeros_like(rest)
    for t in range(T):
        pos[tets[t, 1:]] = F[t].T
    E = np.full(T, 1e5)
    cpu = scenes._assemble(name="degenerate", pos_rest=rest, pos=pos, vel=np.zeros_like(pos), tets=tets, E=E, nu=0.45,
                           rho=1000.0, dt=0.01, barriers=[])
    _, _, blocks, b = fem.newton_system(rest, pos, np.zeros_like(pos), tets, E, 0.45, 1000.0, 0.01, device=dev)
    got = blocks.cpu().numpy()[:10 * T].reshape(T, 90)
    ref = cpu.blocks[:10 * T].reshape(T, 90)
    mu, lam = 1e5 / 2.9, 1e5 * 0.45 / (1.45 * 0.1)
    f = np.linalg.norm(F, axis=(1, 2))
    scale = 1e-4 / 6.0 * 12.0 * (mu + lam * f ** 4 + lam * (f ** 3 + 2.0) * f)
    assert (np.abs(got - ref).max(axis=1) <= 1e-12 * scale).all()
    np.testing.assert_allclose(b.cpu().numpy(), cpu.b, atol=1e-12 * T * np.abs(cpu.b).max())
