"""The single-precision PM adjoint on either side of the grid size up to which its
solve runs beside the density's: against the double-precision one (another chain
of transforms), and what the device holds for it."""
import numpy as np
import pytest

import hsr
import synth
from hsr_testutil import force_errors

pytestmark = pytest.mark.gpu

TOL = (3e-5, 2e-3)  # single precision, as the adjoint's other tests


def _inputs(ng, n=20000):
    p = synth.random_box(n, float(ng + 9), ng)
    return p, np.random.default_rng(ng).standard_normal((n, 3)).astype(np.float32)


@pytest.mark.parametrize("ng", [256, 512, 520])
def test_either_form(ctx, ng):
    p, u = _inputs(ng)
    got, want = (ctx.pm_vjp(p.x, p.y, p.z, u, hsr.pm_params(ng, 4, 1.0, 0.7, 0.3, prec))
                 for prec in (hsr.PM_F32, hsr.PM_F64))
    rms, mx = force_errors(got, want)
    assert rms <= TOL[0] and mx <= TOL[1], (rms, mx)
    # the grids are the forward kick's again
    v = [np.zeros(p.n, np.float32) for _ in range(6)]
    prm = hsr.pm_params(ng, 4, 1.0, 0.7, 0.3, hsr.PM_F32)
    ctx.pm_kick(p.x, p.y, p.z, *v[:3], prm)
    with hsr.Context() as fresh:
        fresh.pm_kick(p.x, p.y, p.z, *v[3:], prm)
    rms, mx = force_errors(np.stack(v[:3], 1), np.stack(v[3:], 1))
    assert rms <= TOL[0] and mx <= TOL[1], (rms, mx)


def test_large_grids_hold_the_deposits_only(hsr_lib):
    torch = pytest.importorskip("torch")
    ng = 540
    p, u = _inputs(ng)
    prm = hsr.pm_params(ng, 4, 1.0, 1.0, 1.0, hsr.PM_F32)
    with hsr.Context() as ctx:
        ctx.pm_kick(p.x, p.y, p.z, *[np.zeros(p.n, np.float32) for _ in range(3)], prm)
        free = torch.cuda.mem_get_info()[0]
        ctx.pm_vjp(p.x, p.y, p.z, u, prm)
        # the three deposited fields, 12 bytes a cell, and a third for plans
        assert free - torch.cuda.mem_get_info()[0] <= 16 * ng**3
