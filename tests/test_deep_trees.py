"""Trees deeper than a subtree block's bookkeeping holds (48 levels below its
root), which the device build makes again level by level: the host build's
permutation and lists, bit for bit, on a context whose buffers hold what larger
trees of other shapes left there, and on a fresh one.

Masses growing threefold along a line put the centre of mass between the last
two particles, so every split takes one particle off."""
import numpy as np
import pytest

import hsr
import synth

pytestmark = pytest.mark.gpu


def _set(n, line, first):
    """n particles of mass 1 in a box, and a line beside it."""
    rng = np.random.default_rng(n + line)
    x = (rng.random((n, 3)) * 20 + (10, 0, 0)).astype(np.float32)
    q = np.full((line, 3), 3.0, np.float32)
    q[:, 0] = 1 + 0.125 * np.arange(line)
    x = np.concatenate([x, q])
    m = np.concatenate([np.ones(n), first * 3.0 ** np.arange(line)]).astype(np.float32)
    n += line
    return synth.Particles(*(np.ascontiguousarray(x[:, d]) for d in range(3)),
                           *rng.standard_normal((3, n)).astype(np.float32), m,
                           np.zeros(n, np.float32), np.arange(n, dtype=np.int64),
                           np.zeros(n, np.uint16), nglt=(30, 30, 30))


def _compare(ctx, p, nd=1):
    kp = synth.kick_params(p, nd=nd, fcoeff=0.0)
    # the leaves of a corner: the tree is compared whole
    kp.min_force, kp.max_force = (0.5,) * 3, (5.0,) * 3
    q = p.copy()
    host = hsr.HostLists(q, kp)
    ctx.rcb_kick(p, kp)
    for k in ("x", "y", "z", "mass", "id"):
        assert np.array_equal(getattr(p, k).view(np.uint8), getattr(q, k).view(np.uint8)), k
    assert ctx.stats()["processed_leaves"] == host.nleaves > 0
    for a, b in zip(ctx.lists(), host.get()):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))


# 48 particles of a line reach level 47, the deepest a block holds; 70 reach 69
@pytest.mark.parametrize("n,line,first", [(0, 48, 1.0), (0, 49, 1.0), (0, 70, 1.0),
                                          (100, 70, 1e-35), (20000, 70, 1e-35)])
def test_deep_tree_after_another(hsr_lib, n, line, first):
    ctx = hsr.Context()
    try:
        _compare(ctx, _set(n, line, first))        # nothing there yet
        _compare(ctx, _set(40000, 1, 1.0))         # several roots, levels 0 to about 20
        _compare(ctx, _set(n, line, first))        # what it left is there
        _compare(ctx, _set(9000, 1, 1.0))
    finally:
        ctx.close()


def test_more_than_64_levels_of_large_nodes(ctx):
    """Masses growing by exp(70) along a line of 200,000: 68 levels of nodes too
    large for a subtree block, each with centres of mass to certify, 77 in all."""
    n = 200_000
    x = np.full((n, 3), 3.0, np.float32)
    x[:, 0] = 1 + 0.125 * np.arange(n)
    z = np.zeros((4, n), np.float32)
    p = synth.Particles(*(np.ascontiguousarray(x[:, d]) for d in range(3)), *z[:3],
                        np.exp(70.0 * np.arange(n) / n).astype(np.float32), z[3],
                        np.arange(n, dtype=np.int64), np.zeros(n, np.uint16), nglt=(25001, 4, 4))
    _compare(ctx, p, nd=64)
