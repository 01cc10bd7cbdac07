"""The device tree's centre-of-mass sums over sets whose masses are not all the
same, or not of ordinary size, and nodes that are not split, against the host
build: the same permutation of every array, bit for bit, and the same lists."""
import numpy as np
import pytest

import hsr
import synth

pytestmark = pytest.mark.gpu


def same_bits(a, b):
    return np.array_equal(a.view(np.uint8), b.view(np.uint8))


def same_or_nan(a, b):  # (NaN has other bits on each machine)
    return np.array_equal(a, b, equal_nan=a.dtype == np.float32)


def compare(ctx, x, mass, nd, lists=4, same=same_bits, **opening):
    """The tree whole, the lists of the leaves in a corner; the kick's statistics."""
    n = len(x)
    zero = np.zeros((4, n), np.float32)
    p = synth.Particles(*(np.ascontiguousarray(x[:, d], np.float32) for d in range(3)), *zero[:3],
                        np.asarray(mass, np.float32), zero[3], np.arange(n, dtype=np.int64),
                        np.zeros(n, np.uint16), nglt=(int(np.ceil(x.max())) + 1,) * 3)
    kp = synth.kick_params(p, nd=nd, fcoeff=0.0, **opening)
    corner = float(np.quantile(x, 0.3))
    kp.min_force, kp.max_force = (-1.0,) * 3, (corner,) * 3
    q = p.copy()
    host = hsr.HostLists(q, kp)
    stats = ctx.rcb_kick(p, kp)
    for k in ("x", "y", "z", "mass", "id"):
        assert np.array_equal(getattr(p, k).view(np.uint8), getattr(q, k).view(np.uint8)), k
    assert stats["processed_leaves"] == host.nleaves
    if host.nleaves:
        for a, b in zip(ctx.lists()[:lists], host.get()):
            assert same(a, b)
    return stats


@pytest.mark.parametrize("n", [40, 3000, 8192, 9000, 70000])
def test_one_magnitude_of_both_signs(ctx, n):
    rng = np.random.default_rng(n)
    x = (rng.random((n, 3)) * 20).astype(np.float32)
    compare(ctx, x, np.where(rng.random(n) < 0.1, -1.0, 1.0), 8)


@pytest.mark.parametrize("n", [40, 3000, 9000])
def test_one_mass_of_more_bits_than_the_sums_hold(ctx, n):
    """A mass near the smallest normal numbers, whose last bits lie below the
    sums' last place, on a lattice coarse enough that the terms' do not."""
    rng = np.random.default_rng(n)
    x = 256.0 * rng.integers(1, 17, (n, 3))
    compare(ctx, x, np.full(n, (1 + 2.0**-20) * 2.0**-112), 8)


def _heavy(rng, n, factor):  # one particle that outweighs the rest
    m = np.ones(n, np.float32)
    m[n // 3] = factor
    return m


def _spread(rng, n, factor):
    return (factor ** rng.random(n)).astype(np.float32)


def _species(rng, n, factor):
    return np.where(rng.random(n) < 0.5, np.float32(1), np.float32(factor))


# ranges on both sides of the one from which the sums take the third integer,
# and beyond what that holds; with a far particle, masses of one value too
@pytest.mark.parametrize("make,factor,far", [
    (_heavy, 2.0**11, None), (_heavy, 2.0**12, None), (_heavy, 1e6, None), (_heavy, 1e-6, None),
    (_heavy, 1e9, None), (_heavy, 1e15, None), (_spread, 1e4, None), (_spread, 1e8, None),
    (_species, 1e6, None), (_heavy, 1.0, 1e4), (_heavy, 1.0, 1e9), (_heavy, 1.0, -1e9),
    (_heavy, 1e6, 1e6), (_heavy, 0.0, None)])
@pytest.mark.parametrize("n,nd", [(3000, 4), (30000, 16), (300000, 64)])
def test_sets_of_wide_range(ctx, n, nd, make, factor, far):
    rng = np.random.default_rng(n)
    x = (rng.random((n, 3)) * 30).astype(np.float32)
    if far is not None:
        x[n // 2, 1] = far
    st = compare(ctx, x, make(rng, n, factor), nd)
    # what the third integer holds is decided without the sequential sums: by 40
    # in a thousand nodes' three quotients at most, 2^-31 of a term's range a term
    # against the 2^-25 that a quotient is rounded by
    if make is _heavy and 1e6 <= max(factor, abs(far or 0)) <= 1e9:
        assert st["cm_fallbacks"] <= 0.04 * st["nodes"]


@pytest.mark.parametrize("n,nd", [(30000, 9000), (30000, 40000), (70000, 20000)])
def test_leaves_larger_than_a_subtree_block(ctx, n, nd):
    rng = np.random.default_rng(n + nd)
    compare(ctx, (rng.random((n, 3)) * 20).astype(np.float32), np.ones(n), nd)


@pytest.mark.parametrize("n", [300, 9000])
def test_one_place(ctx, n):
    """Every split leaves a part empty: the root is the only leaf, above its size."""
    compare(ctx, np.full((n, 3), 0.1, np.float32), np.ones(n), 16)


def _massless(nd, share):
    rng = np.random.default_rng(nd)
    x = (rng.random((3001, 3)) * 20).astype(np.float32)
    return x, np.where(rng.random(3001) < share, 0.0, 1.0), nd


MASSLESS = [(1, 1, 0.1), (2, 1, 0.5), (8, 1, 0.1), (8, 1, 1.2), (2, 12, 0.5)]


@pytest.mark.parametrize("share", [0.2, 0.7])
@pytest.mark.parametrize("nd,tdpts,angle", MASSLESS)
def test_lists_with_massless_nodes(ctx, nd, tdpts, angle, share):
    """Nodes whose particles have no mass have no centre of mass (NaN): no test
    of a distance from it holds, the one that drops far nodes neither."""
    compare(ctx, *_massless(nd, share), lists=3, tdpts=tdpts, open_angle=angle)


@pytest.mark.parametrize("axes", [(2,), (1, 2), (0,)])
def test_flat_sets(ctx, axes):
    """Axes a thousandth as long as the others: their terms, too, keep the bits
    that decide the centres of mass (one in a few hundred nodes went to the
    sequential sums)."""
    n = 500_000
    x = np.random.default_rng(4).random((n, 3)) * 100
    x[:, axes] *= 1e-3
    st = compare(ctx, x.astype(np.float32), np.ones(n), 64)
    assert st["cm_fallbacks"] <= 5e-4 * st["nodes"]
