"""The device list walk (a warp per leaf over windows of its stack) against the
host build: the same leaves and the same entries in the same order, where a
leaf has more segments than the walk's per-leaf region, where trees are deep or
uneven, and where whole nodes are taken as pseudo-particles."""
import numpy as np
import pytest

import hsr
import synth

pytestmark = pytest.mark.gpu

CASES = [
    ("one leaf", lambda: synth.random_box(40, 6.0, 1), 64, 1, 0.1),
    ("two leaves", lambda: synth.random_box(65, 6.0, 2), 64, 1, 0.1),
    ("33 leaves' segments", lambda: synth.random_box(900, 9.0, 3), 32, 1, 0.1),
    ("over 256 segments a leaf", lambda: synth.random_box(3000, 9.0, 4), 2, 1, 0.1),
    ("leaf size 1", lambda: synth.random_box(1500, 12.0, 5), 1, 1, 0.5),
    ("wide angle, monopole", lambda: synth.random_box(6000, 14.0, 6), 8, 1, 1.2),
    ("wide angle, 12-point", lambda: synth.random_box(6000, 14.0, 6), 8, 12, 1.0),
    ("clustered", lambda: synth.clustered_box(16, nhalo=3, seed=7), 16, 1, 0.1),
    ("line", lambda: synth.sorted_line(5000), 16, 1, 0.1),
]


@pytest.mark.parametrize("make,nd,tdpts,angle", [c[1:] for c in CASES], ids=[c[0] for c in CASES])
def test_lists_in_the_host_builds_order(ctx, make, nd, tdpts, angle):
    p = make()
    kp = synth.kick_params(p, nd=nd, tdpts=tdpts, open_angle=angle, fcoeff=1.0)
    kp.min_force, kp.max_force = (0.2,) * 3, tuple(float(g) for g in p.nglt)
    q = p.copy()
    host = hsr.HostLists(q, kp)
    ctx.rcb_kick(p, kp)
    assert ctx.stats()["processed_leaves"] == host.nleaves > 0
    for a, b in zip(ctx.lists(), host.get()):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    # pseudo-particles (n and above) go by each build's own node numbers
    a, b = ctx.lists_index(), host.index()
    assert np.array_equal(np.minimum(a, p.n), np.minimum(b, p.n))


def test_lists_launched_ahead_of_their_sizes(hsr_lib):
    """One context over sets that do and do not fit the buffers of the call
    before: more entries, fewer, the same entries in more work items, and lists
    that need the second walk; each call's lists as the host builds them."""
    ctx = hsr.Context()
    try:
        for n, side, nd, group in ((900, 9.0, 32, 32), (6000, 14.0, 16, 32), (900, 9.0, 32, 32),
                                   (6000, 14.0, 64, 32), (6000, 14.0, 64, 16), (3000, 9.0, 2, 16),
                                   (6000, 14.0, 16, 16), (1, 9.0, 32, 32), (6000, 14.0, 64, 16)):
            ctx.set_tune("batched", 128, group)
            p = synth.random_box(n, side, n + nd)
            kp = synth.kick_params(p, nd=nd, fcoeff=1.0)
            kp.min_force, kp.max_force = (0.2,) * 3, tuple(float(g) for g in p.nglt)
            q, v = p.copy(), p.copy()
            host = hsr.HostLists(q, kp)
            ctx.rcb_kick(p, kp)
            for a, b in zip(ctx.lists(), host.get()):
                assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), (n, nd, group)
            fresh = hsr.Context()
            fresh.set_tune("batched", 128, group)
            fresh.rcb_kick(v, kp)
            assert fresh.stats()["work_items"] == ctx.stats()["work_items"]
            assert np.array_equal(p.vx, v.vx) and np.array_equal(p.id, v.id)
            fresh.close()
    finally:
        ctx.close()
