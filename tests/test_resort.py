"""The sort by cell inside the device sub-cycle, bit for bit against the
oracle's restatement of Particles::map1 and resortParticles, where its two
forms begin and end: cells up to and above the longest one whose ranks are
counted (1024), grids of more than eight cells a particle, runs of 32
out-of-box particles, sets of one particle.  The kick's coefficient is zero,
so that velocities are only permuted and every array must come out equal."""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu

G = 12


def _set(rng, n, dense=0, outside=0):
    u = rng.uniform(0, G, (n, 3)).astype(np.float32)
    u = np.minimum(u, np.nextafter(np.float32(G), np.float32(0)))
    if dense:  # exactly `dense` particles in one cell
        u[np.all(np.floor(u) == (5, 6, 7), axis=1)] += 1.0
        u[rng.permutation(n)[:dense]] = (np.float32([5, 6, 7]) +
                                         rng.uniform(0.1, 0.9, (dense, 3)).astype(np.float32))
    if outside:  # scattered over the index range, some of it far away
        far = np.float32([-0.25, G, 300.0, -1e30, 1e30])
        at = rng.permutation(n)[:outside]
        u[at, rng.integers(0, 3, outside)] = far[rng.integers(0, 5, outside)]
    v = rng.normal(0, 1, (3, n)).astype(np.float32)
    return synth.Particles(*(np.ascontiguousarray(u[:, d]) for d in range(3)), *v,
                           rng.uniform(1, 2, n).astype(np.float32),
                           rng.normal(0, 1, n).astype(np.float32),
                           np.arange(n, dtype=np.int64), np.arange(n).astype(np.uint16),
                           nglt=(G, G, G))


@pytest.mark.parametrize("stream", [False, True])
@pytest.mark.parametrize("n,dense,outside", [
    (1, 0, 0), (31, 0, 0), (215, 0, 9), (216, 0, 9), (4097, 0, 700), (6000, 32, 0), (6000, 33, 65),
    (6000, 1024, 40), (6000, 1025, 40), (3000, 0, 3000)])
def test_sort_by_cell(ctx, oracle_lib, n, dense, outside, stream):
    p = _set(np.random.default_rng(n + 7 * dense + outside), n, dense, outside)
    ts = synth.stepper(z_in=50.0, z_fin=10.0, nsteps=10).advanced(1)
    kp = synth.kick_params(p, nd=64, fcoeff=0.0)
    q = p.copy()
    _, nin = ctx.subcycle(p, kp, 1, p.nglt, ts.alpha, ts.pp, float(synth.stream_tau(ts, 1)), ts.adot,
                          skip_stream=not stream)
    want = oracle_lib.subcycle(q, ts, 1, kp, stream=stream, fcoeff=0.0)
    assert nin == want
    if not stream:
        assert nin == n - outside
    for k in synth.FIELDS:
        assert np.array_equal(getattr(p, k).view(np.uint8), getattr(q, k).view(np.uint8)), k
