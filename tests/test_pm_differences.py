"""The PM solve's gradient as 4th-order differences of one inverse transform
(double precision), and their transpose in the adjoint, at the grid sizes where
the wrap and the kernels' tiles can go wrong, against the restatement."""
import numpy as np
import pytest

import hsr
import pm_oracle
import synth
from hsr_testutil import force_errors

pytestmark = pytest.mark.gpu


def _particles(ng, ngo, seed):
    p = synth.random_box(6 * ng ** 2 + 40, float(ng + 2 * ngo + 1), seed)
    u = np.random.default_rng(seed + 1).standard_normal((p.n, 3)).astype(np.float32)
    return p, u


@pytest.mark.parametrize("ng", [2, 4, 6, 16, 18, 34, 66])
def test_gradient_fields(ctx, ng):
    ngo = 1 if ng < 6 else 4
    p, _ = _particles(ng, ngo, ng)
    rho, grad = ctx.pm_fields(p.x, p.y, p.z, hsr.pm_params(ng, ngo))
    want_rho, want = pm_oracle.fields(p.x, p.y, p.z, ng, ngo)
    if ng == 2:  # every difference wraps onto itself
        assert np.abs(grad).max() == 0.0
        return
    rms, mx = force_errors(grad.reshape(3, -1).T, want.reshape(3, -1).T)
    assert rms <= 1e-5 and mx <= 1e-3, (rms, mx)


@pytest.mark.parametrize("ng", [4, 6, 18, 34])
@pytest.mark.parametrize("precision,tol", [(hsr.PM_F64, (1e-5, 1e-3)), (hsr.PM_F32, (3e-5, 2e-3))])
def test_adjoint(ctx, ng, precision, tol):
    ngo = 1 if ng < 6 else 4
    p, u = _particles(ng, ngo, 100 + ng)
    got = ctx.pm_vjp(p.x, p.y, p.z, u, hsr.pm_params(ng, ngo, 1.0, 0.7, 0.3, precision))
    want = 0.7 * 0.3 * pm_oracle.vjp64(p.x, p.y, p.z, u, ng, ngo)
    rms, mx = force_errors(got, want)
    assert rms <= tol[0] and mx <= tol[1], (rms, mx)
