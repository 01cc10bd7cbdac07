"""Positions that are not finite: the device build makes the host build's
permutation, its groups hold every particle of a leaf once whatever the
coordinates' order, and the next call on the context is not affected."""
import numpy as np
import pytest

import hsr
import synth

pytestmark = pytest.mark.gpu


def _set(n, values, seed):
    p = synth.random_box(n, 8.0, seed)
    rng = np.random.default_rng(seed)
    at = rng.permutation(n)[:max(1, n // 10)]
    for i, a in enumerate(at):
        (p.x, p.y, p.z)[rng.integers(0, 3)][a] = values[i % len(values)]
    return p


def _params(p, nd):
    kp = synth.kick_params(p, nd=nd, fcoeff=0.5)
    kp.min_force, kp.max_force = (-1.0,) * 3, (9.0,) * 3
    return kp


@pytest.mark.parametrize("values", [(np.nan,), (np.inf,), (-np.inf,), (np.inf, np.nan, -np.inf), (3e38,)],
                         ids=["nan", "inf", "-inf", "all", "huge"])
@pytest.mark.parametrize("n,nd", [(12, 64), (20, 64), (33, 64), (40, 8), (200, 256), (256, 8), (700, 8),
                                  (3000, 64), (9000, 64)])
def test_permutation_groups_and_the_next_call(ctx, n, nd, values):
    p = _set(n, values, n + nd)
    kp = _params(p, nd)
    q, f = p.copy(), p.copy()
    hsr.HostLists(q, kp)
    ctx.rcb_kick(p, kp)
    for k in ("x", "y", "z", "mass", "id"):
        assert np.array_equal(getattr(p, k).view(np.uint8), getattr(q, k).view(np.uint8)), k
    # a tape's groups are ordered in halves
    ctx.force_fwd(f.x, f.y, f.z, f.mass, kp)
    ctx.force_vjp(np.ones((n, 3), np.float32))
    a = synth.random_box(100, 6.0, 1)
    b = a.copy()
    ctx.rcb_kick(a, _params(a, 32))
    with hsr.Context() as fresh:
        fresh.rcb_kick(b, _params(b, 32))
    assert np.array_equal(a.id, b.id) and np.array_equal(a.vx, b.vx)
