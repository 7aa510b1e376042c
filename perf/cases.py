"""Performance cases: the calls that one implicit-Euler Newton iteration makes.

A simulator that uses this framework does the following in every Newton iteration, and each of
the calls is a case kind here:

* ``fem``      Hessian producer: triplets and gradient of a tet mesh (``FemScene.assemble``);
* ``contact``  barrier gradients and Hessians of the contact pairs (``contact.barrier``);
* ``solve``    triplets to Newton direction: convert, MAS build / assembly, PCG
               (``Solver.solve_linear_system``), FP64 and FP32, both bank sizes, both
               preconditioners, with and without contacts;
* ``batch``    the same for many uneven scenes in one solve (``ConcatenatedBatch.solve``);
* ``ccd``      the line search's step bound over the swept pairs (``ccd.step_size``);
* ``energy``   the line search's incremental potential (``FemScene.energy``).

Scenes are seeded versions of the benchmark configurations: a jittered cube of n^3 hexes (6 tets
each) falling onto a ground barrier, the heterogeneous cube squashed by a slab (per-tet Young's
modulus log-uniform in [1e4, 1e8] Pa over Voronoi regions), two stacked cubes in contact, and
two facing sheets for the pair kernels.  The inputs and the FP64 references (``exact``) are plain
numpy / torch; the framework is only called in ``prepare`` (handles) and ``run``.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "stiff-gipc_b200"))

from stgipc import PCGSolverConfig, Solver  # noqa: E402
from stgipc import ccd, contact  # noqa: E402
from stgipc.batch import ConcatenatedBatch  # noqa: E402
from stgipc.fem import FemScene  # noqa: E402
from stgipc.scenes import NewtonSystem  # noqa: E402

DEV = "cuda"
NU, RHO, DT, GY = 0.45, 1000.0, 1.0 / 60.0, -9.8
DHAT, KAPPA = 1e-3, 1e5            # ground and slab barriers
PAIR_DHAT, PAIR_KAPPA = 1e-6, 1e5  # squared activation distance of the contact pairs


# ---------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------
def _solve(n, scene="cube", precision="fp64", bank=16, precond="mas", stop="reference"):
    return dict(kind="solve", n=n, scene=scene, precision=precision, bank=bank, precond=precond, stop=stop)


def listed():
    rel = "relative_residual"
    return [
        # a few hundred vertices: launches and host round trips, as in a small interactive scene
        dict(_solve(6), name="solve-cube6"),
        # the default configuration (FP64, MAS, reference stop rule): 14,739 DOF
        dict(_solve(16), name="solve-cube16"),
        # two cubes in contact, contact triplets and pairs in the system, the FP32 path
        dict(_solve(13, scene="stack", precision="fp32", stop=rel), name="solve-stack13-fp32"),
        # 32-vertex banks, an odd vertex count, strong stiffness contrast
        dict(_solve(22, scene="het", bank=32, stop=rel), name="solve-het22-bank32"),
        # the headline system (352,947 DOF) in both precisions
        dict(_solve(48, scene="het", precision="fp32", stop=rel), name="solve-het48-fp32"),
        dict(_solve(48, scene="het", stop=rel), name="solve-het48-fp64"),
        # many uneven scenes as one system with per-scene recurrences
        dict(kind="batch", count=48, n_hi=12, precision="fp32", name="batch48-fp32"),
        # the Hessian producer on the default and on the headline mesh
        dict(kind="fem", n=16, scene="cube", name="fem-cube16"),
        dict(kind="fem", n=48, scene="het", name="fem-het48"),
        # one evaluation of the line search's potential (180k tets)
        dict(kind="energy", n=31, scene="het", name="energy-het31"),
        # contact pairs of a draped cloth on a solid
        dict(kind="contact", pairs=30001, name="contact-30k"),
        # swept pairs of a surface step
        dict(kind="ccd", pairs=100003, per_pair=False, name="ccd-100k"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    k = rng.random()
    if k < 0.5:
        precond = "diag" if rng.random() < 0.15 else "mas"
        scene = rng.choice(["cube", "het", "het", "stack"])
        hi = 20 if precond == "diag" else (24 if scene == "stack" else 48)
        return _solve(log(4, hi), scene, rng.choice(["fp64", "fp32"]), rng.choice([16, 16, 16, 32]), precond,
                      rng.choice(["reference", "relative_residual"]))
    if k < 0.58:
        return dict(kind="batch", count=rng.randint(5, 60), n_hi=rng.randint(5, 12),
                    precision=rng.choice(["fp64", "fp32"]))
    if k < 0.72:
        return dict(kind="fem", n=log(4, 48), scene=rng.choice(["cube", "het"]))
    if k < 0.80:
        return dict(kind="energy", n=log(4, 48), scene=rng.choice(["cube", "het"]))
    if k < 0.90:
        return dict(kind="contact", pairs=log(200, 300000))
    return dict(kind="ccd", pairs=log(500, 400000), per_pair=rng.random() < 0.5)


# ---------------------------------------------------------------------------------------
# meshes
# ---------------------------------------------------------------------------------------
def _spread(v):
    """The low 10 bits of v, three apart."""
    out = np.zeros_like(v)
    for b in range(10):
        out |= ((v >> b) & 1) << (3 * b)
    return out


def _csr(V, tets):
    e = np.concatenate([tets[:, [a, b]] for a in range(4) for b in range(a + 1, 4)])
    key = np.unique(np.concatenate([e[:, 0] * V + e[:, 1], e[:, 1] * V + e[:, 0]]))
    src, dst = key // V, key % V
    num = np.bincount(src, minlength=V)
    start = np.concatenate([[0], np.cumsum(num)[:-1]])
    return start.astype(np.uint32), num.astype(np.uint32), dst.astype(np.uint32)


@functools.lru_cache(maxsize=16)
def _grid(n):
    """(vertices, tets, neighbour lists) of the unit cube of n^3 hexes split into six tets
    along the main diagonal, vertices in Morton order."""
    m = n + 1
    z, y, x = (a.ravel() for a in np.meshgrid(*[np.arange(m)] * 3, indexing="ij"))
    pos = np.stack([x, y, z], 1) / n
    k, j, i = (a.ravel() for a in np.meshgrid(*[np.arange(n)] * 3, indexing="ij"))
    tets = []
    for p in ((0, 1, 2), (1, 2, 0), (2, 0, 1), (0, 2, 1), (2, 1, 0), (1, 0, 2)):
        c = np.stack([i, j, k], 1)
        vs = [c]
        for ax in p:
            c = c.copy()
            c[:, ax] += 1
            vs.append(c)
        v = [c[:, 0] + m * (c[:, 1] + m * c[:, 2]) for c in vs]
        odd = p in ((0, 2, 1), (2, 1, 0), (1, 0, 2))
        tets.append(np.stack([v[0], v[2], v[1], v[3]] if odd else v, 1))
    tets = np.stack(tets, 1).reshape(-1, 4)
    q = np.minimum(pos * 1024, 1023).astype(np.int64)
    order = np.argsort(_spread(q[:, 0]) * 4 + _spread(q[:, 1]) * 2 + _spread(q[:, 2]), kind="stable")
    new = np.empty_like(order)
    new[order] = np.arange(order.size)
    tets = new[tets]
    return pos[order], tets, _csr(m ** 3, tets)


def _slots(V, bank):
    M = -(-V // bank) * bank
    pm = np.full(M, -1, np.int32)
    pm[:V] = np.arange(V)
    return pm, np.arange(V, dtype=np.int32)


def _state(n, scene, seed):
    """Scene state (the FemScene layout) of a falling or a squashed heterogeneous cube."""
    rng = np.random.default_rng(seed)
    grid, tets, _ = _grid(n)
    jit = 0.05 / n
    if scene == "het":
        rest = grid + rng.uniform(-jit, jit, grid.shape)
        sites = rng.uniform(0.0, 1.0, (8, 3))
        site_E = np.exp(rng.uniform(math.log(1e4), math.log(1e8), 8))
        cent = rest[tets].mean(axis=1)
        E = site_E[np.argmin(np.stack([((cent - s) ** 2).sum(1) for s in sites], 1), axis=1)]
        y = rest[:, 1]
        pos = rest.copy()
        pos[:, 1] -= 0.08 * y * y * (1.0 + 0.3 * np.sin(np.pi * rest[:, 0]) * np.sin(np.pi * rest[:, 2]))
        pos[:, 0] += 0.0016 * (rest[:, 0] - 0.5) * y
        pos[:, 2] += 0.0016 * (rest[:, 2] - 0.5) * y
        pos += rng.uniform(-0.05 * jit, 0.05 * jit, pos.shape)
        pos[:, 1] += 4e-4 - pos[:, 1].min()
        vel = np.zeros_like(pos)
        vel[:, 1] = -rest[:, 1]
        planes = [((0.0, 1.0, 0.0), 0.0, DHAT, KAPPA), ((0.0, -1.0, 0.0), -(pos[:, 1].max() + 4e-4), DHAT, KAPPA)]
    else:
        rest = grid + np.array([0.0, 5e-4, 0.0]) + rng.uniform(-jit, jit, grid.shape)
        rest[grid[:, 1] == 0.0, 1] = 5e-4
        # mid-step: a smooth deformation with local noise, as Newton meets it
        pos = rest + 2e-2 * np.sin(3.0 * rest[:, [1, 2, 0]]) * rest[:, 1:2] + rng.uniform(-0.1 * jit, 0.1 * jit, grid.shape)
        pos[:, 1] = np.maximum(pos[:, 1], 4e-4)
        E = np.full(tets.shape[0], 1e5)
        vel = np.zeros_like(pos)
        vel[:, 1] = -2.0
        planes = [((0.0, 1.0, 0.0), 0.0, DHAT, KAPPA)]
    return dict(pos_rest=rest, pos=pos, vel=vel, tets=tets, E=E, nu=NU, rho=RHO, dt=DT, barriers=planes)


def _stack_state(n, seed):
    """Two cubes, the upper one shifted by a fraction of a cell and a small gap above the
    lower one; also the point-triangle pairs between the facing layers."""
    a, b = _state(n, "cube", seed), _state(n, "cube", seed + 7919)
    rng = np.random.default_rng(seed + 104729)
    V = a["pos"].shape[0]
    grid = _grid(n)[0]
    h = 1.0 / n
    for s in (a, b):  # flat facing layers
        s["pos"] = s["pos_rest"].copy()
        s["pos_rest"][grid[:, 1] == 1.0, 1] = 1.0005
        s["pos"][:, 1] = s["pos_rest"][:, 1]
    a["pos"][grid[:, 1] == 0.0, 1] = 5e-4
    b["pos"] = b["pos"] + np.array([0.6 * h, 1.0, 0.3 * h])
    low = grid[:, 1] == 0.0
    b["pos"][low, 1] = 1.0005 + rng.uniform(1e-4, 8e-4, int(low.sum()))
    b["pos_rest"] = b["pos_rest"] + np.array([0.6 * h, 1.0, 0.3 * h])
    state = dict(a)
    for k in ("pos_rest", "pos", "vel", "E"):
        state[k] = np.concatenate([a[k], b[k]])
    state["tets"] = np.concatenate([a["tets"], b["tets"] + V])
    at = {tuple(c): v for v, c in enumerate(np.rint(grid * n).astype(int))}
    pairs = [(-(at[i, 0, k] + V) - 1, at[i, n, k], at[i + 1, n, k], at[i + 1, n, k + 1])
             for i in range(n) for k in range(n)]
    return state, np.array(pairs, np.int32)


# ---------------------------------------------------------------------------------------
# the Newton system in plain torch (FP64)
# ---------------------------------------------------------------------------------------
def _cof(F):
    return torch.stack([torch.linalg.cross(F[:, 1], F[:, 2]), torch.linalg.cross(F[:, 2], F[:, 0]),
                        torch.linalg.cross(F[:, 0], F[:, 1])], 1)


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV).to(dtype)


def _scatter(idx, val, V):
    """[V, 3] sums of val [.., 3] over the vertices idx, in index order (the inputs have to be
    the same bits every time they are made)."""
    i, v = idx.reshape(-1).cpu().numpy(), val.reshape(-1, 3).cpu().numpy()
    return _t(np.stack([np.bincount(i, v[:, k], V) for k in range(3)], 1))


def _kinematics(s):
    rest, pos, tets = _t(s["pos_rest"]), _t(s["pos"]), _t(s["tets"], torch.int64)
    Dm = (rest[tets[:, 1:]] - rest[tets[:, :1]]).transpose(1, 2)
    Ds = (pos[tets[:, 1:]] - pos[tets[:, :1]]).transpose(1, 2)
    det = (Dm[:, :, 0] * torch.linalg.cross(Dm[:, :, 1], Dm[:, :, 2])).sum(1)
    Di = _cof(Dm).transpose(1, 2) / det[:, None, None]
    E = _t(s["E"])
    mu, lam = E / (2.0 * (1.0 + NU)), E * NU / ((1.0 + NU) * (1.0 - 2.0 * NU))
    F = Ds @ Di
    g = _cof(F)
    J = (F[:, 0] * g[:, 0]).sum(1)
    vol = det.abs() / 6.0
    mass = _scatter(tets, (RHO * vol / 4.0)[:, None, None].expand(-1, 4, 3), rest.shape[0])[:, 0].contiguous()
    return pos, tets, Di, F, g, J, vol, mu, lam, mass


def _plane_terms(s, pos):
    """(gradient [V, 3], Hessian [V, 3, 3], energy [V]) of the barrier planes."""
    V = pos.shape[0]
    G = torch.zeros(V, 3, dtype=torch.float64, device=DEV)
    H = torch.zeros(V, 3, 3, dtype=torch.float64, device=DEV)
    e = torch.zeros(V, dtype=torch.float64, device=DEV)
    for nrm, off, dhat, kappa in s["barriers"]:
        nv = torch.tensor(nrm, dtype=torch.float64, device=DEV)
        d = pos @ nv - off
        on = d < dhat
        d2 = torch.where(on, d * d, torch.full_like(d, dhat * dhat))
        t, lg = d2 - dhat * dhat, torch.log(d2 / (dhat * dhat))
        gb = -2.0 * t * lg - t * t / d2
        hb = -2.0 * lg - 4.0 * t / d2 + t * t / (d2 * d2)
        z = torch.zeros_like(d)
        G += torch.where(on, kappa * gb * 2.0 * d, z)[:, None] * nv
        H += torch.where(on, kappa * (4.0 * hb * d2 + 2.0 * gb), z)[:, None, None] * torch.outer(nv, nv)
        e += torch.where(on, -kappa * t * t * lg, z)
    return G, H, e


def _newton_system(s):
    """(rows, cols, blocks [N, 9] column-major, b) of the implicit-Euler Newton iteration at
    pos: 10 upper blocks per tet, then one diagonal block per vertex."""
    pos, tets, Di, F, g, J, vol, mu, lam, mass = _kinematics(s)
    T, V = tets.shape[0], pos.shape[0]
    k = lam * (J - 1.0 - mu / lam)
    eps = torch.zeros(3, 3, 3, dtype=torch.float64, device=DEV)
    for i, j, l in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
        eps[i, j, l], eps[i, l, j] = 1.0, -1.0
    HJ = torch.einsum("ikm,jln,tmn->tijkl", eps, eps, F).reshape(T, 9, 9)
    gv = g.reshape(T, 9)
    H = k[:, None, None] * HJ
    H += lam[:, None, None] * gv[:, :, None] * gv[:, None, :]
    H.diagonal(dim1=1, dim2=2).add_(mu[:, None])
    for Hc in H.split(1 << 14):
        w, Q = torch.linalg.eigh(Hc)
        Hc.copy_(torch.where((w < 0).any(1)[:, None, None], (Q * w.clamp_min(0.0)[:, None, :]) @ Q.mT, Hc))
    P = mu[:, None] * F.reshape(T, 9) + k[:, None] * gv
    d = torch.cat([-Di.sum(1, keepdim=True), Di], 1)  # [T, 4, 3]
    wt = vol * DT * DT
    f = wt[:, None, None] * (d @ P.reshape(T, 3, 3).mT)
    half = torch.einsum("taj,tijkl->taikl", d, H.reshape(T, 3, 3, 3, 3))
    full = wt[:, None, None, None, None] * torch.einsum("tbl,taikl->tabik", d, half)
    rows, cols, blocks = [], [], []
    for a in range(4):
        for b in range(a, 4):
            r, c = tets[:, a], tets[:, b]
            sw = r > c
            B = full[:, a, b]
            rows.append(torch.where(sw, c, r))
            cols.append(torch.where(sw, r, c))
            blocks.append(torch.where(sw[:, None, None], B, B.mT))  # column-major storage
    G, Hp, _ = _plane_terms(s, pos)
    vel = _t(s["vel"])
    grad = mass[:, None] * (-DT * vel - DT * DT * torch.tensor([0.0, GY, 0.0], dtype=torch.float64, device=DEV)) + G
    grad += _scatter(tets, f, V)
    Hp.diagonal(dim1=1, dim2=2).add_(mass[:, None])
    vid = torch.arange(V, device=DEV)
    rows = torch.cat([torch.stack(rows, 1).reshape(-1), vid]).to(torch.int32)
    cols = torch.cat([torch.stack(cols, 1).reshape(-1), vid]).to(torch.int32)
    blocks = torch.cat([torch.stack(blocks, 1).reshape(-1, 9), Hp.reshape(-1, 9)])
    return rows, cols, blocks, grad.reshape(-1)


def _decode(pairs):
    """(type, vertex ids [P, 4]) of sign-encoded pairs; 0 PP, 1 PE, 2 PT, 3 EE."""
    q = pairs.long()
    ee = q[:, 0] >= 0
    typ = torch.where(ee, 3, torch.where(q[:, 2] < 0, 0, torch.where(q[:, 3] < 0, 1, 2)))
    vid = q.clone()
    vid[:, 0] = torch.where(ee, q[:, 0], -q[:, 0] - 1)
    return typ, vid


def _pair_terms(pairs, x):
    """(gradient [P, 12], blocks [P, 10, 9]) of the pair barriers, zero where inactive."""
    typ, vid = _decode(pairs)
    v = x[vid.clamp_min(0)].detach().requires_grad_(True)
    a, b, c, d = v.unbind(1)
    dot = lambda p, q: (p * q).sum(1)  # noqa: E731
    cr = torch.linalg.cross
    pe, pt, ee = cr(b - a, c - a), cr(c - b, d - b), cr(b - a, d - c)
    one = torch.ones_like(a[:, 0])
    safe = lambda q, m: torch.where(m, q, one)  # noqa: E731
    m = [typ == k for k in range(4)]
    d2 = torch.where(m[0], dot(a - b, a - b), torch.where(
        m[1], dot(pe, pe) / safe(dot(c - b, c - b), m[1]), torch.where(
            m[2], dot(a - b, pt) ** 2 / safe(dot(pt, pt), m[2]), dot(c - a, ee) ** 2 / safe(dot(ee, ee), m[3]))))
    s = torch.sqrt(d2) / math.sqrt(PAIR_DHAT)
    h = torch.autograd.grad(s.sum(), v)[0].reshape(-1, 12)
    s = s.detach()
    scale = 4.0 * PAIR_KAPPA * PAIR_DHAT ** 2
    I, lI = s * s, torch.log(s * s)
    e1 = torch.where(s < 1.0, s * scale * lI * (I - 1.0) * (I + I * lI - 1.0) / I, 0.0)
    I = I.clamp_min(1e-6)
    lI = torch.log(I)
    e2 = -scale * (4 * I + lI - 3 * I * I * lI * lI + 6 * I * lI - 2 * I * I + I * lI * lI - 7 * I * I * lI - 2) / I
    e2 = torch.where(s < 1.0, e2, 0.0)
    cnt = typ.clamp_max(2) + 2
    blocks = []
    for i in range(4):
        for j in range(i, 4):
            B = e2[:, None, None] * h[:, 3 * i:3 * i + 3, None] * h[:, None, 3 * j:3 * j + 3]
            B = torch.where((vid[:, i] > vid[:, j])[:, None, None], B, B.mT)
            blocks.append(torch.where((j < cnt)[:, None, None], B, 0.0).reshape(-1, 9))
    return e1[:, None] * h, torch.stack(blocks, 1), typ, vid


def _solve_system(case, seed):
    """(rows, cols, blocks, b, contacts or None, vertex count, neighbour lists)."""
    n = case["n"]
    start, num, nlist = _grid(n)[2]
    V = (n + 1) ** 3
    if case["scene"] != "stack":
        return _newton_system(_state(n, case["scene"], seed)) + (None, V, (start, num, nlist))
    s, pairs = _stack_state(n, seed)
    rows, cols, blocks, b = _newton_system(s)
    pairs = _t(pairs, torch.int32)
    G, H, _, vid = _pair_terms(pairs, _t(s["pos"]))
    ij = [(i, j) for i in range(4) for j in range(i, 4)]
    r = torch.stack([torch.minimum(vid[:, i], vid[:, j]) for i, j in ij], 1).reshape(-1).to(torch.int32)
    c = torch.stack([torch.maximum(vid[:, i], vid[:, j]) for i, j in ij], 1).reshape(-1).to(torch.int32)
    b = b + _scatter(vid, G, 2 * V).reshape(-1)
    nb = (np.concatenate([start, start + nlist.size]), np.concatenate([num, num]), np.concatenate([nlist, nlist + V]))
    return torch.cat([rows, r]), torch.cat([cols, c]), torch.cat([blocks, H.reshape(-1, 9)]), b, pairs, 2 * V, nb


def _batch_systems(case, seed):
    """NewtonSystem objects of uneven cubes, n log-uniform in [3, n_hi]; the sizes are the
    case's own, the states the seed's."""
    rs, rng = np.random.default_rng(case["count"] * 1000 + case["n_hi"]), np.random.default_rng(seed)
    ns = [int(round(math.exp(rs.uniform(math.log(3), math.log(case["n_hi"]))))) for _ in range(case["count"])]
    states = [_state(n, "cube", int(rng.integers(1 << 30))) for n in ns]
    voff = np.concatenate([[0], np.cumsum([(n + 1) ** 3 for n in ns])])
    toff = np.concatenate([[0], np.cumsum([6 * n ** 3 for n in ns])])
    cat = dict(states[0])
    for k in ("pos_rest", "pos", "vel"):
        cat[k] = np.concatenate([s[k] for s in states])
    cat["E"] = np.concatenate([s["E"] * math.exp(rng.uniform(math.log(0.1), math.log(100.0))) for s in states])
    cat["tets"] = np.concatenate([s["tets"] + o for s, o in zip(states, voff)])
    rows, cols, blocks, b = (a.cpu().numpy() for a in _newton_system(cat))
    out = []
    for k, n in enumerate(ns):
        v0, v1, t0, t1 = voff[k], voff[k + 1], 10 * toff[k], 10 * toff[k + 1]
        d0 = 10 * toff[-1] + v0
        pick = lambda a: np.concatenate([a[t0:t1], a[d0:d0 + v1 - v0]])  # noqa: E731,B023
        st, nm, nl = _grid(n)[2]
        out.append(NewtonSystem(f"cube{n}", int(v1 - v0), (pick(rows) - v0).astype(np.int32),
                                (pick(cols) - v0).astype(np.int32), pick(blocks), b[3 * v0:3 * v1].copy(),
                                states[k]["pos"], states[k]["tets"], st, nm, nl, np.zeros((0, 4), np.int32)))
    return out, (rows, cols, blocks, b)


# ---------------------------------------------------------------------------------------
# two facing sheets: contact pairs and swept pairs
# ---------------------------------------------------------------------------------------
def _sheets(pairs, h, gap, seed):
    """Lower and upper m x m vertex grids of pitch h, the upper one shifted by (0.6, 0.3) h and
    gap (lo, hi) above; (x [2 m^2, 3], cell indices of half the pairs, m, rng)."""
    rng = np.random.default_rng(seed)
    half = -(-pairs // 2)
    m = int(math.ceil(math.sqrt(half))) + 3
    i, k = (a.ravel() for a in np.meshgrid(np.arange(m), np.arange(m), indexing="ij"))
    low = np.stack([i * h, 0.0 * i, k * h], 1) + rng.uniform(-0.02 * h, 0.02 * h, (m * m, 3)) * [1, 0, 1]
    up = np.stack([(i + 0.6) * h, rng.uniform(*gap, m * m), (k + 0.3) * h], 1)
    up += rng.uniform(-0.02 * h, 0.02 * h, (m * m, 3)) * [1, 0, 1]
    c = np.arange(half)
    return np.concatenate([low, up]), (1 + c // (m - 3), 1 + c % (m - 3)), m, rng


def _contact_pairs(case, seed):
    P = case["pairs"]
    x, (i, k), m, rng = _sheets(P, 1.2e-3, (5e-5, 7e-4), seed)
    L, U = (lambda a, b: a * m + b), (lambda a, b: m * m + a * m + b)
    neg = np.full_like(i, -1)
    pt = np.stack([-U(i, k) - 1, L(i, k), L(i + 1, k), L(i + 1, k + 1)], 1)
    pe = np.stack([-U(i, k) - 1, L(i, k), L(i + 1, k + 1), neg], 1)
    pp = np.stack([-U(i, k) - 1, L(i + 1, k), neg, neg], 1)
    t = rng.random(i.size)[:, None]
    first = np.where(t < 0.7, pt, np.where(t < 0.85, pe, pp))
    ee = np.stack([U(i, k), U(i + 1, k), L(i + 1, k), L(i + 1, k + 1)], 1)
    return np.concatenate([first, ee])[:P].astype(np.int32), x


def _swept_pairs(case, seed):
    P, h = case["pairs"], 1e-2
    x, (i, k), m, rng = _sheets(P, h, (2e-3, 2e-2), seed)
    L, U = (lambda a, b: a * m + b), (lambda a, b: m * m + a * m + b)
    di, dk = rng.integers(-1, 2, (2, i.size))
    a, b = i + di, k + dk
    other = rng.random(i.size)[:, None] < 0.5
    tri = np.where(other, np.stack([L(a, b), L(a + 1, b), L(a + 1, b + 1)], 1),
                   np.stack([L(a, b), L(a + 1, b + 1), L(a, b + 1)], 1))
    pt = np.concatenate([(-U(i, k) - 1)[:, None], tri], 1)
    ee = np.stack([U(i, k), U(i + 1, k), L(a + 1, b), L(a + 1, b + 1)], 1)
    dx = rng.normal(0.0, 2e-4, x.shape)
    dx[m * m:, 1] -= rng.uniform(0.0, 1.5e-2, m * m)
    return np.concatenate([pt, ee])[:P].astype(np.int32), x, dx


# ---------------------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        rows, cols, blocks, b, contacts, V, nb = _solve_system(case, seed)
        solver = Solver(PCGSolverConfig(bank_size=case["bank"], precision=case["precision"],
                                        preconditioner=case["precond"], stop_rule=case["stop"]))
        if case["precond"] == "mas":
            solver.mas_init(V, *nb, *_slots(V, case["bank"]))
        torch.cuda.synchronize()
        return dict(kind=kind, solver=solver, rows=rows, cols=cols, blocks=blocks.reshape(-1), b=b,
                    x=torch.zeros_like(b), contacts=contacts)
    if kind == "batch":
        systems, _ = _batch_systems(case, seed)
        return dict(kind=kind, batch=ConcatenatedBatch(systems, PCGSolverConfig(precision=case["precision"]), device=DEV))
    if kind in ("fem", "energy"):
        scene = FemScene(_state(case["n"], case["scene"], seed), gravity_y=GY, device=DEV)
        g = torch.tensor([0.0, GY, 0.0], dtype=torch.float64, device=DEV)
        xtilde = (scene.pos + DT * scene.vel + DT * DT * g).contiguous()
        return dict(kind=kind, scene=scene, x=scene.pos.clone(), xtilde=xtilde)
    if kind == "contact":
        pairs, x = _contact_pairs(case, seed)
        return dict(kind=kind, pairs=_t(pairs, torch.int32), x=_t(x))
    pairs, x, dx = _swept_pairs(case, seed)
    return dict(kind=kind, pairs=_t(pairs, torch.int32), x=_t(x), dx=_t(dx), per_pair=case["per_pair"])


def run(s):
    kind = s["kind"]
    if kind == "solve":
        s["solver"].solve_linear_system(s["rows"], s["cols"], s["blocks"], s["b"], s["x"], contacts=s["contacts"])
        return s["x"]
    if kind == "batch":
        s["batch"].solve()
        return s["batch"].x
    if kind == "fem":
        sc = s["scene"]
        sc.assemble(s["x"], s["xtilde"])
        return sc.rows, sc.cols, sc.blocks, sc.b
    if kind == "energy":
        return s["scene"].energy(s["x"], s["xtilde"])
    if kind == "contact":
        return contact.barrier(s["pairs"], s["x"], PAIR_DHAT, PAIR_KAPPA)
    return ccd.step_size(s["pairs"], s["x"], s["dx"], slackness=0.8, per_pair=s["per_pair"])


# ---------------------------------------------------------------------------------------
# work and 64-bit references
# ---------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("solve", "batch"):
        # triplets, b and x once, the neighbour lists once; a product with the merged upper
        # blocks (7.8 a vertex) for the residual.  The iterations' own traffic comes on top.
        if kind == "solve":
            scenes, copies = [case["n"]], 2 if case["scene"] == "stack" else 1
        else:
            rs, copies = np.random.default_rng(case["count"] * 1000 + case["n_hi"]), 1
            scenes = [int(round(math.exp(rs.uniform(math.log(3), math.log(case["n_hi"]))))) for _ in range(case["count"])]
        T = copies * sum(6 * n ** 3 for n in scenes)
        V = copies * sum((n + 1) ** 3 for n in scenes)
        return dict(bytes=80.0 * (10 * T + V) + 48.0 * V + 60.0 * V + 80.0 * 7.8 * V, flops=90.0 * T + 36.0 * 7.8 * V)
    if kind in ("fem", "energy"):
        T, V = 6 * case["n"] ** 3, (case["n"] + 1) ** 3
        if kind == "energy":
            return dict(bytes=24.0 * T + 72.0 * V, flops=250.0 * T + 30.0 * V)
        return dict(bytes=24.0 * T + 72.0 * V + 80.0 * (10 * T + V) + 24.0 * V, flops=8000.0 * T + 60.0 * V)
    P = case["pairs"]
    V = 2 * (math.ceil(math.sqrt(-(-P // 2))) + 3) ** 2
    if kind == "contact":
        return dict(bytes=16.0 * P + 24.0 * V + 896.0 * P, flops=800.0 * P)
    return dict(bytes=16.0 * P + 48.0 * V + (8.0 * P if case["per_pair"] else 8.0), flops=4000.0 * P)


def _direct(rows, cols, blocks, b):
    """A x = b from upper 3x3 triplets: block-Jacobi CG in FP64, restarted until the true
    residual stops falling."""
    rows, cols, V = rows.long(), cols.long(), b.numel() // 3
    key, inv = torch.unique(rows * V + cols, return_inverse=True)
    B = torch.zeros(key.numel(), 9, dtype=torch.float64, device=DEV).index_add_(0, inv, blocks.reshape(-1, 9))
    B = B.view(-1, 3, 3).mT  # row-major
    r, c = key // V, key % V
    D = torch.zeros(V, 3, 3, dtype=torch.float64, device=DEV)
    D[r[r == c]] = B[r == c]
    Dinv = torch.linalg.inv(D)
    off = r != c
    r, c, B = torch.cat([r, c[off]]), torch.cat([c, r[off]]), torch.cat([B, B[off].mT])
    o = torch.arange(3, device=DEV)
    ri = (3 * r[:, None, None] + o[None, :, None]).expand(-1, 3, 3).reshape(-1)
    ci = (3 * c[:, None, None] + o[None, None, :]).expand(-1, 3, 3).reshape(-1)
    order = torch.argsort(ri * (3 * V) + ci)
    ptr = torch.zeros(3 * V + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.bincount(ri, minlength=3 * V).cumsum(0)
    A = torch.sparse_csr_tensor(ptr, ci[order], B.reshape(-1)[order], (3 * V, 3 * V))
    pre = lambda v: (Dinv @ v.view(V, 3, 1)).reshape(-1)  # noqa: E731
    x, last = torch.zeros_like(b), float("inf")
    for _ in range(4):
        res = b - A @ x
        norm = float(res.norm() / b.norm())
        if norm < 1e-14 or norm > 0.3 * last:
            break
        last = norm
        z = pre(res)
        p, rz, goal = z.clone(), res @ z, 1e-10 * float(res.norm())
        for it in range(20000):
            q = A @ p
            al = rz / (p @ q)
            x = x + al * p
            res = res - al * q
            if it % 64 == 63 and float(res.norm()) <= goal:
                break
            z = pre(res)
            new = res @ z
            p = z + (new / rz) * p
            rz = new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        rows, cols, blocks, b = _solve_system(case, seed)[:4]
        return _direct(rows, cols, blocks, b)
    if kind == "batch":
        systems, _ = _batch_systems(case, seed)
        voff = np.concatenate([[0], np.cumsum([s.num_verts for s in systems])])
        rows = np.concatenate([s.rows + o for s, o in zip(systems, voff)])
        cols = np.concatenate([s.cols + o for s, o in zip(systems, voff)])
        return _direct(_t(rows, torch.int64), _t(cols, torch.int64), _t(np.concatenate([s.blocks for s in systems])),
                       _t(np.concatenate([s.b for s in systems])))
    if kind == "fem":
        _, _, blocks, b = _newton_system(_state(case["n"], case["scene"], seed))
        return None, None, blocks.reshape(-1), b
    if kind == "energy":
        s = _state(case["n"], case["scene"], seed)
        pos, tets, Di, F, g, J, vol, mu, lam, mass = _kinematics(s)
        psi = 0.5 * mu * ((F * F).sum((1, 2)) - 3.0) + 0.5 * lam * (J - 1.0 - mu / lam) ** 2
        step = DT * _t(s["vel"]) + DT * DT * torch.tensor([0.0, GY, 0.0], dtype=torch.float64, device=DEV)
        e = (vol * DT * DT * psi).sum() + 0.5 * (mass * (step * step).sum(1)).sum() + _plane_terms(s, pos)[2].sum()
        return float(e), None
    if kind == "contact":
        pairs, x = _contact_pairs(case, seed)
        G, H, _, _ = _pair_terms(_t(pairs, torch.int32), _t(x))
        return None, None, H.reshape(-1, 9), G, None
    return None
