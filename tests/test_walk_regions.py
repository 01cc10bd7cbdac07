"""The list walk's per-leaf regions where there are too many leaves for full
ones (a leaf size of 1): what the device holds for them stays bounded, and the
leaves that do not fit theirs come out as the host builds them."""
import numpy as np
import pytest

import hsr
import synth

pytestmark = pytest.mark.gpu


def test_two_million_leaves(hsr_lib):
    torch = pytest.importorskip("torch")
    n = 2_000_000  # 33 segments a region; 600 to 2100 entries a list
    p = synth.random_box(n, 50.0, 1)
    kp = synth.kick_params(p, nd=1, fcoeff=0.0)
    kp.min_force, kp.max_force = (0.0,) * 3, (2.0,) * 3
    q = p.copy()
    host = hsr.HostLists(q, kp)
    ctx = hsr.Context()
    try:
        small = synth.random_box(100, 6.0, 2)
        ctx.rcb_kick(small, synth.kick_params(small))
        free = torch.cuda.mem_get_info()[0]
        ctx.rcb_kick(p, kp)
        used = free - torch.cuda.mem_get_info()[0]
        assert np.array_equal(p.id, q.id)
        for a, b in zip(ctx.lists(), host.get()):
            assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
        # 512 MB of regions and a quarter to grow, about 950 bytes a particle else
        assert used < 1.25 * 2**29 + 1200 * n, used
    finally:
        ctx.close()
