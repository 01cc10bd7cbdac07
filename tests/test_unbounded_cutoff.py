"""The 5th-order law without a cutoff (its fsrrmax infinite, or beyond every
distance): the entries and particles that fill up the pair kernels' lanes stay
out of the sums.  Against the dense sum over pairs in FP64, at odd list lengths
and group sizes.

Tolerance, in units of u = 2^-24 against the sum S of the absolute values of
all terms: y = rsqrt(s) within 5 u (s by 5 u, the approximation by 2.5 u), its
fifth power within 30 u with the products; weights, cotangents and polynomials
15 u, in the forward kernel's powers of s = r2 + 0.01 as well; a sum of at most
50 values 50 u.  100 u covers them."""
import numpy as np
import pytest

import hsr
import synth

pytestmark = pytest.mark.gpu

COEF = np.float64(np.float32((0.269327, -0.0750978, 0.0114808, -0.00109313, 0.0000605491,
                              -0.00000147177)))
RSM = float(np.float32(0.1))
FCOEFF = float(np.float32(0.7))


def _terms(x):
    d = x[None] - x[:, None]  # [i, j]: x_j - x_i
    r2 = (d * d).sum(2)
    y = 1 / np.sqrt(r2 + RSM * RSM)
    k = np.arange(6)
    pw, dpw = r2[..., None] ** k, k[1:] * r2[..., None] ** (k[1:] - 1)
    off = ~np.eye(len(x), dtype=bool)
    return (d, off, y**3 - pw @ COEF, y**3 + pw @ abs(COEF), -1.5 * y**5 - dpw @ COEF[1:],
            1.5 * y**5 + dpw @ abs(COEF[1:]))


def _forward(x, m):
    d, off, g, gabs, _, _ = _terms(x)
    w = np.where(off, FCOEFF * m[None], 0.0)
    return ((w * g)[..., None] * d).sum(1), ((w * gabs)[..., None] * abs(d)).sum(1)


def _gradient(x, m, u):
    d, off, g, gabs, dg, dgabs = _terms(x)
    w = np.where(off, FCOEFF * m[None], 0.0)[..., None]
    v = w * (g[..., None] * u[:, None] + 2 * (dg * (d * u[:, None]).sum(2))[..., None] * d)
    vabs = w * (gabs[..., None] * abs(u[:, None])
                + 2 * (dgabs * (abs(d) * abs(u[:, None])).sum(2))[..., None] * abs(d))
    return v.sum(0) - v.sum(1), vabs.sum(0) + vabs.sum(1)


def _set(n):
    rng = np.random.default_rng(n)
    return (rng.uniform(1.0, 4.0, (n, 3)).astype(np.float32),
            rng.uniform(0.5, 2.0, n).astype(np.float32),
            rng.standard_normal((n, 3)).astype(np.float32))


@pytest.mark.parametrize("fsrrmax", [np.inf, 3e18, 1e15])
@pytest.mark.parametrize("n", [1, 7, 16, 33, 45])
def test_callers_lists(hsr_lib, n, fsrrmax):
    torch = pytest.importorskip("torch")
    x, m, _ = _set(n)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    v = [torch.zeros(n, device="cuda") for _ in range(3)]
    hsr.kick_lists_noalloc(dev(np.concatenate([x, m[:, None]], 1)), n, dev(np.int32([0])),
                           dev(np.int32([n])), dev(np.int64([0])), dev(np.int32([n])),
                           dev(np.arange(n, dtype=np.int32)), *v, FCOEFF, RSM, fsrrmax, 1)
    want, scale = _forward(x.astype(np.float64), m.astype(np.float64))
    got = torch.stack(v, 1).cpu().numpy()
    assert np.all(np.abs(got - want) <= 100 * 2.0**-24 * scale)


@pytest.mark.parametrize("fsrrmax", [np.inf, 3e18, 1e15])
@pytest.mark.parametrize("n", [1, 7, 16, 33, 45])
def test_force_and_gradient(ctx, n, fsrrmax):
    x, m, u = _set(n)
    p = synth.Particles(*(np.ascontiguousarray(x[:, d]) for d in range(3)), *np.zeros((3, n), np.float32),
                        m, np.zeros(n, np.float32), np.arange(n, dtype=np.int64),
                        np.zeros(n, np.uint16), nglt=(5, 5, 5))
    kp = synth.kick_params(p, nd=64, fcoeff=FCOEFF, open_angle=0.0, rsm=RSM)
    kp.min_force, kp.max_force, kp.law, kp.fsrrmax = (0.0,) * 3, (5.0,) * 3, 1, fsrrmax
    force = ctx.force_fwd(p.x, p.y, p.z, p.mass, kp)
    got = ctx.force_vjp(u)
    times = len(ctx.lists_index()) // n  # a tree of one leaf lists it twice
    assert np.all(np.bincount(ctx.lists_index(), minlength=n) == times)
    x, m, u = (a.astype(np.float64) for a in (x, m, u))
    want, scale = _forward(x, m)
    assert np.all(np.abs(force - times * want) <= 100 * 2.0**-24 * times * scale)
    want, scale = _gradient(x, m, u)
    assert np.all(np.abs(got - times * want) <= 100 * 2.0**-24 * times * scale)
