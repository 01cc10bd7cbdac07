"""The device tree build where its forms begin and end -- a subtree block's
8192 elements, the chunk sizes' 4, 8 and 16 elements a thread, levels of more
than 512 nodes inside a subtree, the two-integer sums' truncated and mixed
terms -- against the host build: the same permutation of every array, bit for
bit, and the same lists."""
import numpy as np
import pytest

import hsr
import synth

pytestmark = pytest.mark.gpu

WAVE = 4 * 152 * 1024  # particles in one wave of 4-element chunks on 152 SMs


def _unit(rng, m):
    return np.ones(m, np.float32)


def _mixed(rng, m):  # 9 decades, all signs of rounding
    return (10.0 ** rng.uniform(-6, 3, m)).astype(np.float32)


def _plain(rng, n, side):
    return (rng.random((n, 3)) * side).astype(np.float32)


def _negative(rng, n, side):
    return _plain(rng, n, side) - np.float32(0.6 * side)


def _ties(rng, n, side):  # equal keys, equal particles
    return np.floor(_plain(rng, n, side))


def _tiny(rng, n, side):  # terms below the sums' last place
    x = _plain(rng, n, side)
    x[rng.random((n, 3)) < 0.3] *= np.float32(1e-25)
    return x


CASES = [
    (0, 8.0, _plain, _unit, 32), (1, 8.0, _plain, _unit, 32), (2, 8.0, _ties, _mixed, 1),
    (255, 9.0, _negative, _mixed, 1), (3000, 12.0, _plain, _mixed, 1), (8191, 20.0, _ties, _unit, 8),
    (8192, 20.0, _negative, _unit, 4), (8193, 20.0, _plain, _mixed, 16), (8193, 20.0, _tiny, _mixed, 3),
    (16385, 25.0, _tiny, _unit, 2), (40000, 30.0, _ties, _mixed, 24), (66000, 30.0, _negative, _mixed, 64),
    (WAVE + 1, 80.0, _plain, _mixed, 300), (2 * WAVE + 1, 100.0, _negative, _unit, 500),
]


@pytest.mark.parametrize("n,side,pos,mass,nd", CASES,
                         ids=[f"{c[0]}{c[2].__name__}{c[3].__name__}" for c in CASES])
def test_permutation_and_lists_are_the_host_builds(ctx, n, side, pos, mass, nd):
    rng = np.random.default_rng(n + nd)
    x = pos(rng, n, side)
    z = lambda: np.zeros(n, np.float32)
    p = synth.Particles(*(np.ascontiguousarray(x[:, d]) for d in range(3)),
                        *rng.standard_normal((3, n)).astype(np.float32), mass(rng, n), z(),
                        np.arange(n, dtype=np.int64), (np.arange(n) % 65521).astype(np.uint16),
                        nglt=(int(side),) * 3)
    kp = synth.kick_params(p, nd=nd, fcoeff=0.0)
    # a corner of the box: the tree is compared whole, the lists of a few leaves
    kp.min_force, kp.max_force = (0.5,) * 3, (4.5,) * 3
    q = p.copy()
    host = hsr.HostLists(q, kp)
    ctx.rcb_kick(p, kp)
    for k in synth.FIELDS:
        if k not in ("vx", "vy", "vz") or n == 0:
            assert np.array_equal(getattr(p, k).view(np.uint8), getattr(q, k).view(np.uint8)), k
    assert ctx.stats()["processed_leaves"] == host.nleaves
    if host.nleaves:
        for a, b in zip(ctx.lists(), host.get()):
            assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
