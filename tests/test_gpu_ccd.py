"""GPU: the CCD step bound (stg_ccd_step_size) against the oracle: every pair's time of
impact and the bound bit for bit (both evaluate the same IEEE operations in the same order;
the device file is compiled without FMA contraction), on random pairs and on the two cubes
in contact pushed into each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _t(a, dev):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def test_random_pairs_bitwise(dev):
    from oracle import oracle as orc
    from stgipc import ccd
    rng = np.random.default_rng(17)
    V = 5000
    x = rng.normal(size=(V, 3))
    dx = rng.normal(size=(V, 3)) * 0.5
    pairs = []
    for i in range(20000):
        v = rng.choice(V, size=4, replace=False)
        pairs.append([-v[0] - 1, v[1], v[2], v[3]] if i % 2 == 0 else list(v))
    pairs = np.array(pairs, np.int32)
    alpha, toc = ccd.step_size(_t(pairs, dev), _t(x, dev), _t(dx, dev), per_pair=True)
    toc = toc.cpu().numpy()
    want = np.array([orc.accd(0 if q[0] < 0 else 1, x[[(-q[0] - 1) if q[0] < 0 else q[0], q[1], q[2], q[3]]],
                              dx[[(-q[0] - 1) if q[0] < 0 else q[0], q[1], q[2], q[3]]], 0.2) for q in pairs])
    assert np.array_equal(toc, want)
    assert (want < 1).sum() > 1000
    assert float(alpha.item()) == orc.ccd_step_size(pairs, x, dx, 0.8)


def test_no_pairs_and_bad_ids(dev):
    import torch
    from stgipc import ccd
    x = _t(np.zeros((4, 3)), dev)
    alpha = ccd.step_size(torch.zeros((0, 4), dtype=torch.int32, device=dev), x, x)
    assert float(alpha.item()) == 1.0
    with pytest.raises(ValueError):
        ccd.step_size(_t(np.array([[-1, 1, 2, 9]], np.int32), dev), x, x)


def test_stacked_cubes_pushed_together(dev):
    """The upper cube moved down by twice the gap: the bound stops it before any pair of the
    interface crosses, and equals the oracle's."""
    from oracle import oracle as orc
    from stgipc import ccd, scenes
    s, _, body = scenes.make_stacked_cubes(8)
    tris = scenes.boundary_faces(s.tets)
    dx = np.zeros_like(s.pos)
    dx[body == 1, 1] = -2e-3
    pairs = scenes.contact_pairs(s.pos, tris, body, dhat=(3e-3) ** 2)
    # CCD pairs: point-triangle and edge-edge only (the reference's _ccd_collisonPairs)
    pt = pairs[(pairs[:, 0] < 0) & (pairs[:, 2] >= 0) & (pairs[:, 3] >= 0)]
    ee = pairs[(pairs[:, 0] >= 0) & (pairs[:, 3] >= 0)]
    cp = np.concatenate([pt, ee])
    assert cp.shape[0] > 100
    alpha = float(ccd.step_size(_t(cp, dev), _t(s.pos, dev), _t(dx, dev)).item())
    assert alpha == orc.ccd_step_size(cp, s.pos, dx, 0.8)
    assert 0.05 < alpha < 0.25   # gap 4e-4 of a 2e-3 push: contact at 0.2
    moved = s.pos + alpha * dx
    for q in cp:
        ids = [(-q[0] - 1) if q[0] < 0 else q[0], q[1], q[2], q[3]]
        d2, _ = orc.contact_d2(2 if q[0] < 0 else 3, moved[ids])
        assert d2 > 0


@pytest.mark.parametrize("P,seed,speed", [(1, 900, 3.0), (31, 902, 0.4), (31, 903, 3.0), (33, 900, 0.4), (33, 901, 3.0),
                                          (129, 902, 0.05), (129, 900, 3.0), (6000, 902, 0.4), (6000, 900, 3.0)])
def test_bound_without_per_pair_times(dev, P, seed, speed):
    """The bound alone stops pairs that cannot lower it: it equals the bound of the full run and
    the oracle's, bit for bit, with degenerate pairs (a zero-length edge, a flat triangle, a
    pair at rest) among them.  The pair that sets it, below one, stands once where it fell and
    once last, in a warp that is not full."""
    from oracle import oracle as orc
    from stgipc import ccd
    rng = np.random.default_rng(seed + P)
    V = 4 * P
    x = rng.normal(size=(V, 3))
    dx = rng.normal(size=(V, 3)) * speed
    v = rng.permutation(V).reshape(P, 4)
    pairs = np.where((np.arange(P) % 2 == 0)[:, None], np.stack([-v[:, 0] - 1, v[:, 1], v[:, 2], v[:, 3]], 1), v).astype(np.int32)
    if P == 1:  # a point on its way through a triangle
        x[v[0]] = [[0.1, 0.5, 0.2], [-1.0, 0.0, -1.0], [1.0, 0.1, -1.0], [0.0, -0.1, 1.0]]
        dx[v[0]] = [[0.0, -0.9, 0.1], [0.0, 0.1, 0.0], [0.1, 0.0, 0.0], [0.0, 0.2, 0.0]]
    for k in range(5, P, 17):
        x[v[k, 3]] = 0.5 * (x[v[k, 1]] + x[v[k, 2]])  # collinear triangle / nearby edge
    for k in range(7, P, 19):
        dx[v[k]] = 0.0
    toc = np.array([orc.accd(0 if q[0] < 0 else 1, x[np.abs(q + (q < 0))], dx[np.abs(q + (q < 0))], 0.2) for q in pairs])
    ok = np.isfinite(toc)
    if not ok.all():
        # the time of a pair that is flat to the last bit is no number: then the bound is none
        for per_pair in (False, True):
            a = ccd.step_size(_t(pairs, dev), _t(x, dev), _t(dx, dev), per_pair=per_pair)
            assert np.isnan(float((a[0] if per_pair else a).item()))
        pairs, toc = pairs[ok], toc[ok]
    want = orc.ccd_step_size(pairs, x, dx, 0.8)
    assert want < 1.0 and want == 1.0 / (1.0 / toc).max()
    k = np.argmin(toc)
    last = np.concatenate([np.delete(pairs, k, 0), pairs[[k]]])
    for p in (pairs, last):
        a0 = ccd.step_size(_t(p, dev), _t(x, dev), _t(dx, dev))
        a1, _ = ccd.step_size(_t(p, dev), _t(x, dev), _t(dx, dev), per_pair=True)
        assert float(a0.item()) == want and float(a1.item()) == want


@pytest.mark.parametrize("P", [33, 6000])
def test_bound_of_regular_pairs_without_per_pair_times(dev, P):
    """As above without degenerate pairs: the bound is a number, set by one pair among many that
    stop early."""
    from oracle import oracle as orc
    from stgipc import ccd
    rng = np.random.default_rng(950 + P)
    V = 4 * P
    x = rng.normal(size=(V, 3))
    dx = rng.normal(size=(V, 3)) * 0.4
    v = rng.permutation(V).reshape(P, 4)
    pairs = np.where((np.arange(P) % 2 == 0)[:, None], np.stack([-v[:, 0] - 1, v[:, 1], v[:, 2], v[:, 3]], 1), v).astype(np.int32)
    a0 = ccd.step_size(_t(pairs, dev), _t(x, dev), _t(dx, dev))
    want = orc.ccd_step_size(pairs, x, dx, 0.8)
    assert want < 1.0 and float(a0.item()) == want


def test_classification_next_to_underflow(dev):
    """Subnormal and zero coordinates beside large ones: the quotients that place the point in a
    region of the triangle underflow.  Every time of impact is the oracle's, bit for bit."""
    from oracle import oracle as orc
    from stgipc import ccd
    h = float.fromhex
    # found by a search on the CPU: the region chosen without dividing gives another last bit
    found = [
        ("0x0p+0 0x0p+0 0x1.536119194736ep+26 0x1.d62b5c7f9c398p+26 0x1.12f5cba6da9f4p+26 -0x0.00000001055a4p-1022 "
         "-0x1.c2522d19258afp+26 -0x1.bf1cd3e951092p+25 0x0p+0 -0x1.1db744f9c0e2ep-1017 -0x1.8f7d4407fc278p-1015 0x0p+0",
         "0x1.1c5361f67dadp+24 0x1.5accfc352095ap+26 -0x1.be6d88d96e42ap+25 -0x1.e08c3d13edbfp+25 0x1.9871b9d4ce89ap+26 "
         "0x1.0491bb7f53174p+26 -0x1.a53667fa657a8p+24 -0x1.53015329351f6p+26 -0x1.8f7a6c1772636p+26 "
         "-0x1.0371156b4b71ap+26 -0x1.4b1368e11cf9ap+26 -0x1.f280d7dc23b1cp+26"),
        ("-0x1.3745845814d7cp+13 0x0p+0 0x1.ba7f5e2e178cp+10 -0x1.da073ebf869e4p+13 -0x1.feb33c6ce785p+11 0x0p+0 "
         "-0x1.d8783aa66f839p+14 0x0p+0 -0x0.0000000002ba5p-1022 0x1.e3116e021be88p+14 -0x0.0000000000a3dp-1022 0x0p+0",
         "0x1.e0d51acdf25f8p+14 -0x1.5f82edbc1e0f4p+14 -0x1.c9e65fa49ebdap+14 -0x1.531534e258a7ep+14 "
         "-0x1.a9be98639fe7ep+13 -0x1.a7e2d9a6acdp+8 0x1.bb5d2de8785bcp+14 -0x1.df7aa65601c94p+14 "
         "-0x1.f04f0f5f0be0dp+14 -0x1.ebf75a5675a9ep+13 0x1.a8bebac0b611p+12 0x1.bcae483989e32p+14"),
        ("0x0p+0 -0x1.5aaa78ee37598p+17 0x1.481f5fdf0300cp+17 0x0p+0 -0x1.6ca2a2186838p+18 0x1.5aea495a6dp+16 "
         "-0x0.0000000000005p-1022 0x0p+0 0x0p+0 0x1.437e12a9e23bp+17 0x0p+0 0x0p+0",
         "0x1.4e675605506bcp+18 -0x1.185c601fa23e8p+18 -0x1.1bd37f3fef346p+17 0x1.280fe1bee2b58p+18 "
         "-0x1.1180049e13b12p+18 -0x1.93dfc7410e808p+18 0x1.812eb28fbeb06p+18 -0x1.11b36b5b9a48p+18 "
         "0x1.f5d76cc7a3b42p+18 -0x1.1b94e4b443d6p+14 0x1.8fdbd937bba36p+18 0x1.7d318503b5a44p+17"),
    ]
    rng = np.random.default_rng(31)
    P = 2000
    s = 2.0 ** rng.integers(0, 30, (P, 1, 1))
    x = rng.uniform(-1, 1, (P, 4, 3)) * s
    kind = rng.integers(0, 6, x.shape)
    x = np.where(kind == 0, 0.0, np.where(kind == 1, np.ldexp(rng.uniform(-1, 1, x.shape), -rng.integers(1000, 1074, x.shape)), x))
    dx = rng.uniform(-1, 1, x.shape) * s
    for k, (a, b) in enumerate(found):
        x[k] = np.array([h(v) for v in a.split()]).reshape(4, 3)
        dx[k] = np.array([h(v) for v in b.split()]).reshape(4, 3)
    q = np.arange(4 * P).reshape(P, 4)
    pairs = np.concatenate([-q[:, :1] - 1, q[:, 1:]], 1).astype(np.int32)
    _, toc = ccd.step_size(_t(pairs, dev), _t(x.reshape(-1, 3), dev), _t(dx.reshape(-1, 3), dev), per_pair=True)
    want = np.array([orc.accd(0, x[k], dx[k], 0.2) for k in range(P)])
    assert (want < 1).sum() > 100
    np.testing.assert_array_equal(toc.cpu().numpy(), want)


def test_early_stop_keeps_a_time_that_falls(dev):
    """A slackness next to one and a thickness: the first step ends within a rounding of the
    thickness, and the second one goes back.  The pair that sets the bound is past the others'
    time after its first step and below it in the end; it comes after them, so that it meets their
    bound.  The bound is the oracle's, with the times and without."""
    from oracle import oracle as orc
    from stgipc import ccd
    h = float.fromhex
    slack, th = 1.0 - 1e-12, 0.5
    # point and triangle, the point's displacement in the pair that sets the bound and in the others
    found = [
        ("0x1.03a5df59f6e6fp-6 -0x1.bfd1f6dccf2e6p-2 0x1.1d11d915932bbp-1 -0x1.e29c51510804ep-1 -0x1.3fef8b51c108cp+0 "
         "0x1.c63f39c94d5bfp-4 0x1.199e8bc1bc4cdp+0 -0x1.019070fb51829p+0 0x1.c70f9635479ecp-5 -0x1.2540078b74c22p-3 "
         "0x1.c3bbbe8eea62fp-1 0x1.696bf7f700514p-8",
         "-0x1.7ce055b124f2bp-26 -0x1.60ba1b06998a8p-25 -0x1.0c249cb28c20bp-20",
         "-0x1.7ce0559e5baa3p-26 -0x1.60ba1af533b24p-25 -0x1.0c249ca55250cp-20"),
        ("0x1.bfb3ca553c5a5p-4 -0x1.cfa6ada15f8c6p-2 0x1.867454d9b1ccbp-2 -0x1.94f7edd5177a2p-1 -0x1.47f3005fd4947p+0 "
         "-0x1.107d9489b7119p-3 0x1.406dc319d65ccp+0 -0x1.a09316ac167a7p-1 -0x1.693d087185b49p-4 -0x1.8c83cf89f68adp-4 "
         "0x1.721c96f949d1ep-1 -0x1.1327b71e80effp-3",
         "0x1.9c69d6f5e3846p-26 -0x1.3404365981961p-27 -0x1.0c58e94e25651p-20",
         "0x1.9c69d6e194047p-26 -0x1.3404364a56454p-27 -0x1.0c58e940ee353p-20"),
    ]
    for v, last, others in found:
        x1 = np.array([h(a) for a in v.split()]).reshape(4, 3)
        x = np.concatenate([x1, x1])
        dx = np.zeros((8, 3))
        dx[0], dx[4] = [h(a) for a in others.split()], [h(a) for a in last.split()]
        t0, t1 = (orc.accd(0, x[4 * k:4 * k + 4], dx[4 * k:4 * k + 4], 1.0 - slack, th) for k in (0, 1))
        assert t1 < t0 < 1.0
        pairs = np.tile(np.array([[-1, 1, 2, 3]], np.int32), (1000000, 1))  # several waves of CTAs
        pairs[-40:] = [-5, 5, 6, 7]
        p = _t(pairs, dev)
        a = ccd.step_size(p, _t(x, dev), _t(dx, dev), slackness=slack, thickness=th)
        b, toc = ccd.step_size(p, _t(x, dev), _t(dx, dev), slackness=slack, thickness=th, per_pair=True)
        assert float(toc[0]) == t0 and float(toc[-1]) == t1
        want = 1.0 / (1.0 / t1)
        assert float(b.item()) == want
        assert float(a.item()) == want
