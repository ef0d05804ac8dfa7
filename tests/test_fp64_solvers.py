"""The FP64 solvers' kernels at the edges of their tiles and lists: the
per-particle walk (bit for bit the oracle's) and the sampled direct sums."""

import numpy as np
import pytest

from native import lopsided_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 63, 65, 129, 1000])
@pytest.mark.parametrize("scale", [1.0, 1e-24, 1e24])
def test_tree_walk_sizes_and_scales_bitwise(ctx, oracle, n, scale):
    """Ragged last warps, lists shorter and longer than a lane's 32 entries,
    and lengths whose squares leave the FP32 range (every test in FP64)."""
    pos, mass = lopsided_sphere(max(n, 8), 4)
    pos, mass = np.ascontiguousarray(pos[:n] * scale), mass[:n].copy()
    kw = dict(G=1.0, theta=0.6, eps=0.02 * scale, quadrupole=True)
    acc, pot = ctx.tree_force(pos, mass, **kw)
    st = ctx.stats()
    want, wpot, (nc, npart) = oracle.tree_force(pos, mass, **kw)
    assert np.array_equal(acc, want, equal_nan=True) and np.array_equal(pot, wpot, equal_nan=True)
    assert (st["cell_interactions"], st["body_interactions"]) == (nc, npart)


@pytest.mark.parametrize("big", [31, 32, 33, 100])
def test_tree_walk_leaf_longer_than_a_list_bitwise(ctx, oracle, big):
    """A leaf of `big` coincident bodies: the lists stop inside it and go on."""
    pos, mass = lopsided_sphere(400, 9)
    pos[:big] = pos[0]
    kw = dict(G=1.7, theta=0.7, eps=0.05, quadrupole=True)
    acc, pot = ctx.tree_force(pos, mass, **kw)
    want, wpot, _ = oracle.tree_force(pos, mass, **kw)
    assert np.array_equal(acc, want) and np.array_equal(pot, wpot)


@pytest.mark.parametrize("quadrupole", [False, True])
@pytest.mark.parametrize("case", ["planar", "line", "window", "massless", "G"])
def test_tree_walk_products_bitwise(ctx, oracle, case, quadrupole):
    """Products worked on the integer pipes: zero components and zero moments
    (with their signs), lengths whose high powers leave the products' window
    for some of a warp's interactions, bodies without mass, G other than 1."""
    pos, mass = lopsided_sphere(2000, 12)
    G, eps = 1.0, 0.01
    if case == "planar":
        pos[:, 2] = 0.0
    elif case == "line":
        pos[:, 1:] = -0.0
    elif case == "window":
        pos, eps = pos * 1e-22, 0.0
    elif case == "massless":
        mass[::3] = 0.0
    else:
        G = 6.674e-11
    kw = dict(G=G, theta=0.6, eps=eps, quadrupole=quadrupole)
    acc, pot = ctx.tree_force(pos, mass, **kw)
    want, wpot, _ = oracle.tree_force(pos, mass, **kw)
    assert np.array_equal(acc, want, equal_nan=True) and np.array_equal(pot, wpot, equal_nan=True)


@pytest.mark.parametrize("n,m", [(1, 1), (127, 5), (128, 128), (129, 129), (3001, 257)])
@pytest.mark.parametrize("scale", [1.0, 1e-160, 1e140])
def test_fp64_sample_sizes_and_scales(ctx, oracle, n, m, scale):
    """Ragged tiles of sources and targets; squared distances far from 1 and
    (the smallest scale) below the normal range. 1e-12 relative, the bound of
    the other sample tests, where the oracle's own squares are normal."""
    import torch
    pos, mass = lopsided_sphere(max(n, 8), 6)
    pos, mass = np.ascontiguousarray(pos[:n] * scale), mass[:n].copy()
    idx = (np.arange(m) * 7 % n).astype(np.uint64)
    kw = dict(G=2.5, eps=0.05 * scale)
    racc, rpot = oracle.direct_fp64(pos, mass, idx=idx, **kw)
    d = lambda a: torch.from_numpy(a).cuda()
    dp, dm, di = d(pos), d(mass), d(idx.astype(np.int64))
    acc = torch.zeros((m, 3), dtype=torch.float64, device="cuda")
    pot = torch.zeros(m, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.direct_fp64_device(dp.data_ptr(), dm.data_ptr(), n, di.data_ptr(), m, acc.data_ptr(),
                           pot.data_ptr(), **kw)
    acc, pot = acc.cpu().numpy(), pot.cpu().numpy()
    if scale == 1e-160:  # r^2 is subnormal in both: a few bits only
        assert np.array_equal(np.isfinite(acc), np.isfinite(racc))
        return
    ok = np.linalg.norm(racc, axis=1) > 0
    err = np.linalg.norm(acc[ok] - racc[ok], axis=1) / np.linalg.norm(racc[ok], axis=1)
    assert err.size == 0 or err.max() < 1e-12
    assert np.all(acc[~ok] == 0)
    assert np.allclose(pot, rpot, rtol=1e-12, atol=0)


def test_fp64_sample_coincident_unsoftened(ctx, oracle):
    """Two bodies at one place without softening: 1/0 gives what it gave."""
    import torch
    pos, mass = lopsided_sphere(300, 2)
    pos[5] = pos[200]
    idx = np.array([5, 7, 200], np.uint64)
    with np.errstate(all="ignore"):
        racc, rpot = oracle.direct_fp64(pos, mass, G=1.0, eps=0.0, idx=idx)
    d = lambda a: torch.from_numpy(a).cuda()
    dp, dm, di = d(pos), d(mass), d(idx.astype(np.int64))
    acc = torch.zeros((3, 3), dtype=torch.float64, device="cuda")
    pot = torch.zeros(3, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.direct_fp64_device(dp.data_ptr(), dm.data_ptr(), 300, di.data_ptr(), 3, acc.data_ptr(),
                           pot.data_ptr(), G=1.0, eps=0.0)
    acc, pot = acc.cpu().numpy(), pot.cpu().numpy()
    assert np.array_equal(np.isnan(acc), np.isnan(racc))
    assert np.array_equal(np.isinf(pot), np.isinf(rpot)) and np.array_equal(pot > 0, rpot > 0)
    assert np.allclose(acc[1], racc[1], rtol=1e-12, atol=0)


@pytest.mark.parametrize("case", ["sheet", "line", "offset", "tiny", "masses", "soft", "hard"])
def test_fp64_sample_fixed_point(ctx, oracle, case):
    """What a tile's fixed point holds and what it does not: a sheet thinner
    than its unit, zero differences, a far offset, coordinates near zero,
    masses that are zero, negative and far apart, softening above and below
    every distance. Each component within 1e-12 of its terms' absolute sum:
    1500 additions and a few roundings a term in both sums, 2^-53 each."""
    import torch
    n = 1500
    pos, mass = lopsided_sphere(n, 21)
    eps = 0.05
    if case == "sheet":
        pos[:, 2] *= 1e-12
    elif case == "line":
        pos[:, 1] = 0.0
        pos[:, 2] = -3.0
    elif case == "offset":
        pos += 1e9
    elif case == "tiny":
        pos[::5] *= 1e-16
    elif case == "masses":
        mass[::3] = 0.0
        mass[1::3] *= -1e-120
        mass[2::9] *= 1e60
    else:
        eps = {"soft": 1e4, "hard": 1e-9}[case]
    idx = (np.arange(140) * 11 % n).astype(np.uint64)
    G = 1.5
    racc, rpot = oracle.direct_fp64(pos, mass, idx=idx, G=G, eps=eps)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dp, dm, di = d(pos), d(mass), d(idx.astype(np.int64))
    acc = torch.zeros((140, 3), dtype=torch.float64, device="cuda")
    pot = torch.zeros(140, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.direct_fp64_device(dp.data_ptr(), dm.data_ptr(), n, di.data_ptr(), 140, acc.data_ptr(),
                           pot.data_ptr(), G=G, eps=eps)
    acc, pot = acc.cpu().numpy(), pot.cpu().numpy()
    dx = pos[idx.astype(np.int64)][:, None, :] - pos[None]
    r2 = (dx * dx).sum(2) + eps * eps
    w = np.where(np.arange(n)[None] == idx[:, None].astype(np.int64), 0.0, 1 / np.sqrt(r2))
    gm = G * np.abs(mass)
    assert np.all(np.abs(acc - racc) <= 1e-12 * np.einsum("tn,tnk->tk", gm * w ** 3, np.abs(dx)))
    assert np.all(np.abs(pot - rpot) <= 1e-12 * (gm * w).sum(1))


def far_cluster(n=20_000):
    """A cube of bodies 8e19 across, seen from a tree of 1e24: the FP32 squares
    of its distances overflow at 1.84e19, their bound on the roundings is 1e18."""
    pos = np.random.default_rng(1).uniform(-4e19, 4e19, (n, 3)) + np.array([2e24, 6e23, -4e23])
    pos[0] *= -1.0
    return pos, np.full(n, 1.0 / n)


@pytest.mark.parametrize("theta", [0.44, 0.45, 0.47])
def test_tree_walk_squares_beyond_fp32_bitwise(ctx, oracle, theta):
    """Cells whose opening distance lies just below sqrt(FLT_MAX), and bodies
    within the roundings of it whose FP32 square is infinite (6 to 28 such pairs
    of a cell to open and a body, by these angles)."""
    pos, mass = far_cluster()
    kw = dict(G=1.0, theta=theta, eps=1e18, quadrupole=True)
    acc, pot = ctx.tree_force(pos, mass, **kw)
    st = ctx.stats()
    want, wpot, (nc, npart) = oracle.tree_force(pos, mass, **kw)
    assert (st["cell_interactions"], st["body_interactions"]) == (nc, npart)
    assert np.array_equal(acc, want) and np.array_equal(pot, wpot)


@pytest.mark.parametrize("warps", [-1, 0])
def test_group_lists_squares_beyond_fp32(gtc, oracle, warps):
    """The same for the grouped walk, by warps and by threads: groups of one body."""
    from checks import compare_lists
    pos, mass = far_cluster()
    kw = dict(theta=0.44, group_size=1, leaf_size=8, pack=False)
    nodes, _, lists = oracle.lists(pos, mass, **kw)
    with gtc.Context(0) as c:
        c.set_option("walk_warps", warps)
        c.group_force(pos, mass, G=1.0, eps=1e18, quadrupole=True, **kw)
        got = c.export()
    assert compare_lists(got, got["nodes"], lists, nodes) == []


@pytest.mark.parametrize("scale", [1e-19, 1e-17, 1e-15, 1e-13, 1e-12, 1e17, 1e18, 1e19, 1e20])
def test_tree_walk_at_the_ends_of_fp32_squares_bitwise(ctx, oracle, scale):
    """Trees of which some tests are within what the FP32 test takes (d^2 from 1e-35
    to 1e38) and some beyond."""
    pos, mass = lopsided_sphere(2000, 15)
    kw = dict(G=1.0, theta=0.6, eps=0.02 * scale, quadrupole=True)
    acc, pot = ctx.tree_force(pos * scale, mass, **kw)
    st = ctx.stats()
    want, wpot, (nc, npart) = oracle.tree_force(pos * scale, mass, **kw)
    assert np.array_equal(acc, want, equal_nan=True) and np.array_equal(pot, wpot, equal_nan=True)
    assert (st["cell_interactions"], st["body_interactions"]) == (nc, npart)
