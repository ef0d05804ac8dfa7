"""The list evaluation at the edges of its tiles: group sizes, list lengths
around a staging round and a slice, softened and not, both ways of sharing a
group's passes, against FP64 sums over the same lists.

Bound: an FP32 sum of L terms in S slices is within (L / S + S) 2^-24 of the sum
of its terms' sizes, and a term (about 20 roundings, rsqrt within 2 ulp)
within 2^-19 of its own: 32 slices and the longest list here (700) give
(700 / 3 + 3 + 32) 2^-24 < 1.7e-5 of the summed sizes.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(T, nc, nb, seed):
    """One group of T targets at the start of 800 bodies, nc cells away from
    them and a body list of its targets and nb others."""
    rng = np.random.default_rng(seed)
    bodies = np.concatenate([rng.uniform(-1, 1, (800, 3)), rng.uniform(0.5, 1, (800, 1))],
                            1).astype(np.float32)
    cells = np.zeros((max(nc, 1), 12), np.float32)
    d = rng.normal(size=(len(cells), 3))
    cells[:, :3] = d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(4, 9, (len(cells), 1))
    cells[:, 3] = rng.uniform(1, 5, len(cells))
    cells[:, 4:10] = rng.uniform(-1, 1, (len(cells), 6))
    cl = rng.permutation(nc).astype(np.uint32)
    bl = rng.permutation(np.concatenate([np.arange(T), T + rng.permutation(800 - T)[:nb]]))
    return bodies, cells, cl, bl.astype(np.uint32)


def _fp64(T, bodies, cells, cl, bl, eps2, quad):
    b, c = bodies.astype(np.float64), cells.astype(np.float64)
    out, size = np.zeros((T, 4)), np.zeros((T, 4))
    for i in range(T):
        def add(t):
            out[i] += t.sum(0)
            size[i] += np.abs(t).sum(0)
        j = bl[bl != i]
        d = b[i, :3] - b[j, :3]
        inv = 1 / np.sqrt((d * d).sum(1) + eps2)
        gm = b[j, 3] * inv
        add(np.concatenate([-(gm * inv * inv)[:, None] * d, -gm[:, None]], 1))
        if len(cl):
            x = c[cl]
            d = b[i, :3] - x[:, :3]
            inv = 1 / np.sqrt((d * d).sum(1) + eps2)
            gm = x[:, 3] * inv
            add(np.concatenate([-(gm * inv * inv)[:, None] * d, -gm[:, None]], 1))
            if quad:
                xx, yy, zz, xy, xz, yz = x[:, 4:10].T
                q = np.stack([xx * d[:, 0] + xy * d[:, 1] + xz * d[:, 2],
                              xy * d[:, 0] + yy * d[:, 1] + yz * d[:, 2],
                              xz * d[:, 0] + yz * d[:, 1] + zz * d[:, 2]], 1)
                rqr = (d * q).sum(1)
                add(np.concatenate([q * (inv ** 5)[:, None]
                                    - 2.5 * (rqr * inv ** 7)[:, None] * d,
                                    -0.5 * (rqr * inv ** 5)[:, None]], 1))
    return out, size


@pytest.mark.parametrize("eps2", [0.0, 1e-30, 1e-3])
@pytest.mark.parametrize("quad", [False, True])
@pytest.mark.parametrize("T", [1, 2, 3, 10, 11, 17, 31, 32])
def test_group_sizes_and_list_lengths(ctx, T, quad, eps2):
    for nc, nb in ((0, 0), (1, 0), (2, 1), (63, 2), (64, 65), (65, 300), (700, 31)):
        bodies, cells, cl, bl = _case(T, nc, nb, 7 * T + nc)
        group = [0, T, 0, len(cl), 0, len(bl), 0, 0]
        G = 0.7
        got = ctx.tree(bodies, cells, cl, bl, np.array([group]), G=G, eps2=eps2,
                       quadrupole=quad)
        want, size = _fp64(T, bodies, cells, cl, bl, np.float64(np.float32(eps2)), quad)
        bound = 1.7e-5 * G * np.linalg.norm(size[:, :3], axis=1)
        assert np.all(np.linalg.norm(got[:T, :3] - G * want[:, :3], axis=1) <= bound), (nc, nb)
        assert np.all(np.abs(got[:T, 3] - G * want[:, 3]) <= 1.7e-5 * G * size[:, 3]), (nc, nb)
        assert np.all(got[T:] == 0)
        # many groups: a warp works a group alone; the same sums bit for bit
        many = ctx.tree(bodies, cells, cl, bl, np.array([group] * 12001), G=G, eps2=eps2,
                        quadrupole=quad)
        assert np.array_equal(got, many), (nc, nb)


def test_small_softening_at_the_origin(ctx):
    """A target at the frame's origin, where the zeros past a list's end lie,
    with a softening whose fifth power underflows: finite and right."""
    bodies = np.array([[0, 0, 0, 1], [1, 0, 0, 2]], np.float32)
    group = np.array([[0, 2, 0, 0, 0, 2, 0, 0]])
    for eps2 in (1e-16, 1e-30):
        got = ctx.tree(bodies, np.zeros((1, 12), np.float32), np.zeros(0, np.uint32),
                       np.arange(2, dtype=np.uint32), group, G=1.0, eps2=eps2)
        assert np.allclose(got, [[2, 0, 0, -2], [-1, 0, 0, -1]], rtol=1e-6, atol=0)


@pytest.mark.parametrize("quad", [False, True])
@pytest.mark.parametrize("eps", [0.0, 0.02])
def test_long_groups_by_teams(gtc, quad, eps):
    """Some 7500 groups, a few of them of bodies far apart with lists many
    times as long: those are worked by teams of warps, the rest by a warp
    each. The same bits as with twice the groups (a warp for every group)."""
    import torch
    rng = np.random.default_rng(3)
    n = 170_000
    pos = rng.normal(size=(n, 3))
    pos *= (rng.random((n, 1)) ** 2 + 1e-3) / np.linalg.norm(pos, axis=1)[:, None]
    pos[:300] = rng.uniform(-2, 2, (300, 3))
    mass = rng.uniform(0.5, 1.5, n) / n
    kw = dict(G=1.0, eps=eps, theta=0.75, quadrupole=quad, leaf_size=8, group_size=32, pack=1)
    with gtc.Context(0) as ctx:
        acc, pot = ctx.group_force(pos, mass, **kw)
        g = ctx.export()["groups"].astype(np.int64)
    assert 6000 <= len(g) < 12000
    work = (g[:, 1] - g[:, 0]) * ((5 if quad else 2) * (g[:, 3] - g[:, 2])
                                  + 2 * (g[:, 5] - g[:, 4]))
    warps = torch.cuda.get_device_properties(0).multi_processor_count * 5 * 4
    assert work.max() > 0.75 * work.sum() / warps
    bufs = []
    with gtc.Ensemble(2) as ens:
        for i in range(2):
            b = [torch.from_numpy(a.copy()).cuda()
                 for a in (pos, np.zeros_like(pos), mass, np.zeros_like(pos), np.zeros(n))]
            bufs.append(b)
            ens.set_system(i, *[t.data_ptr() for t in b], n, **kw)
        ens.set_option("forest", 1)
        torch.cuda.synchronize()
        ens.leapfrog(0.0, 1, prime=True, graph=False)
        torch.cuda.synchronize()
    for b in bufs:
        assert np.array_equal(b[3].cpu().numpy(), acc) and np.array_equal(b[4].cpu().numpy(), pot)
