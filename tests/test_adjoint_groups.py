"""The adjoint pair kernel at the sizes where its split can go wrong: groups
that end inside a half, a pair or a lane's share of pairs, lists that end inside
a batch of 16 entries or a step of 32.  One leaf holds every particle, so the
gradient is the dense sum over pairs, taken in FP64 and over the list as it is
(the walk of a tree that is one leaf lists the leaf twice).

Tolerance, in units of u = 2^-24 against the sum S of the absolute values of
all terms: y = rsqrt(s) is off by 5 u (s by 5 u, the approximation by 2.5 u),
its fifth power by 30 u with the products; weights, cotangents and polynomials
add 15 u; a sum of at most 50 values 50 u.  100 u covers them."""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu

POLY6 = (0.271431, -0.0783394, 0.0133122, -0.00159485, 0.000132336, -0.00000663394, 0.000000147305)
STEP16 = (0.269327, -0.0750978, 0.0114808, -0.00109313, 0.0000605491, -0.00000147177)


def _gradient(x, m, u, times, fcoeff, rsm, rcut, law):
    coef = np.float64(np.float32(STEP16 if law else POLY6))
    d = x[None] - x[:, None]  # [i, j]: x_j - x_i
    r2 = (d * d).sum(2)
    y = 1 / np.sqrt(r2 + rsm * rsm)
    k = np.arange(len(coef))
    pw = r2[..., None] ** k
    dpw = k[1:] * r2[..., None] ** (k[1:] - 1)
    g, gabs = y**3 - pw @ coef, y**3 + pw @ abs(coef)
    dg, dgabs = -1.5 * y**5 - dpw @ coef[1:], 1.5 * y**5 + dpw @ abs(coef[1:])
    off = ~np.eye(len(x), dtype=bool)
    assert not (abs(r2[off] - rcut**2) < 1e-4).any()
    w = np.where(off & (r2 < rcut**2), times * fcoeff * (1 if law else m[:, None]) * m[None], 0.0)
    du = (d * u[:, None]).sum(2)
    v = w[..., None] * (g[..., None] * u[:, None] + 2 * (dg * du)[..., None] * d)
    vabs = w[..., None] * (gabs[..., None] * abs(u[:, None])
                           + 2 * (dgabs * (abs(d) * abs(u[:, None])).sum(2))[..., None] * abs(d))
    return v.sum(0) - v.sum(1), vabs.sum(0) + vabs.sum(1)


@pytest.mark.parametrize("law", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 9, 13, 15, 16, 17, 18, 21, 31, 32, 33, 36, 47, 48, 49])
def test_every_group_size(ctx, n, law):
    rng = np.random.default_rng(100 * n + law)
    x = rng.uniform(2.0, 5.5, (n, 3)).astype(np.float32)
    m = rng.uniform(0.5, 2.0, n).astype(np.float32)
    u = rng.standard_normal((n, 3)).astype(np.float32)
    p = synth.Particles(*(np.ascontiguousarray(x[:, d]) for d in range(3)), *np.zeros((3, n), np.float32),
                        m, np.zeros(n, np.float32), np.arange(n, dtype=np.int64),
                        np.zeros(n, np.uint16), nglt=(8, 8, 8))
    kp = synth.kick_params(p, nd=64, fcoeff=0.7, open_angle=0.0)
    kp.min_force, kp.max_force, kp.law = (0.0,) * 3, (8.0,) * 3, law
    ctx.force_fwd(p.x, p.y, p.z, p.mass, kp)
    got = ctx.force_vjp(u)
    off, cnt, ptr, _ = ctx.lists()
    times = len(ctx.lists_index()) // n
    assert list(cnt) == [n] and np.all(np.bincount(ctx.lists_index(), minlength=n) == times)
    f = lambda v: np.float64(np.float32(v))
    want, scale = _gradient(x.astype(np.float64), m.astype(np.float64), u.astype(np.float64), times,
                            f(0.7), f(kp.rsm), f(kp.fsrrmax), law)
    assert np.all(np.abs(got - want) <= 100 * 2.0**-24 * scale)
