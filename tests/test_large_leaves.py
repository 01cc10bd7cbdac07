"""Leaves too large for one warp to group (more than 256 particles): the kick
over them is right, and grouping them is shared out over the SMs."""
import numpy as np
import pytest

import hsr
import synth
from hsr_testutil import MAX_TOL, RMS_TOL, force_errors, vel

pytestmark = pytest.mark.gpu


def _kick(ctx, p, nd):
    q = p.copy()
    st = ctx.rcb_kick(q, synth.kick_params(p, nd=nd, fcoeff=1.0))
    return q, st


@pytest.mark.parametrize("nd", [257, 512, 1024, 1500])
@pytest.mark.parametrize("group", [16, 32])
def test_kick_and_regroup(hsr_lib, nd, group):
    p = synth.random_box(20000, 14.0, nd)
    p.vx[:] = p.vy[:] = p.vz[:] = 0
    with hsr.Context() as ctx:
        ctx.set_tune("batched", 128, group)
        q, _ = _kick(ctx, p, nd)
        want, _ = _kick(ctx, p, 64)  # another tree of the same particles
        for shape in (48 - group, group):
            ctx.set_tune("batched", 128, shape)  # the groups again, in the other size
            again, _ = _kick(ctx, p, nd)
            rms, mx = force_errors(vel(again), vel(q))
            assert rms <= RMS_TOL and mx <= MAX_TOL
    # (opening angle 0.1: no pseudo-particle within the cutoff at either size)
    a, b = vel(q)[np.argsort(q.id)], vel(want)[np.argsort(want.id)]
    inner = np.all((np.stack([p.x, p.y, p.z], 1) > 5) & (np.stack([p.x, p.y, p.z], 1) < 9), axis=1)
    rms, mx = force_errors(a[inner], b[inner])
    assert rms <= RMS_TOL and mx <= MAX_TOL


def test_time_of_the_lists_does_not_jump(ctx):
    """A set whose leaves are all above 256 particles: lists and groups within ten
    times those of leaves of up to 256 (one block after the other took 30 times)."""
    p = synth.random_box(150000, 30.0, 9)

    def lists_ms(nd):
        return min(_kick(ctx, p, nd)[1]["t_walk_ms"] for _ in range(5))

    assert lists_ms(512) <= 10 * lists_ms(256)
