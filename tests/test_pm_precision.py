"""The double-precision PM solve stays double up to the gradient fields' rounding
to float: against the solver's spectral gradient taken in float64 from the same
density.

Tolerance: half an ulp of the float result, and 1e-12 of the fields' rms for the
differences of the potential -- its float64 rounding, 1e-16 log2(ng) or so of it,
beside a gradient up to ng / 2 pi times smaller: 6e-14 at 130^3 in numpy.  A
potential or a difference in float would be off by 1e-6 and more."""
import numpy as np
import pytest

import hsr
import pm_oracle
import synth

pytestmark = pytest.mark.gpu


def _spectral(rho):
    ng = len(rho)
    _, _, g = pm_oracle.quiet_tables(ng)
    g[0] = g[ng // 2] = 0.0  # both planes' spectra are anti-Hermitian: no real part
    h = ng // 2 + 1
    rk = np.fft.rfftn(rho.astype(np.float64)) * pm_oracle.green(ng)[:, :, :h]
    shapes = [g.reshape(ng, 1, 1), g.reshape(1, ng, 1), g[:h].reshape(1, 1, h)]
    return np.stack([np.fft.irfftn(-1j * s * rk, rho.shape, (0, 1, 2)) * float(ng) ** 3 for s in shapes])


@pytest.mark.parametrize("ng", [4, 18, 66, 130])
@pytest.mark.parametrize("wave", [False, True], ids=["random", "long wave"])
def test_gradient_fields_are_rounded_once(ctx, ng, wave):
    ngo = 1 if ng < 6 else 4
    p = synth.random_box(4 * ng ** 2 + 300, float(ng), ng)
    if wave:  # a density of the box's longest wave along x: the largest potential
        p.x[:] = ng * (p.x / ng) ** np.float32(1.5)
    x, y, z = (np.minimum(a, np.nextafter(np.float32(ng), np.float32(0))) + np.float32(ngo)
               for a in (p.x, p.y, p.z))
    rho, grad = ctx.pm_fields(x, y, z, hsr.pm_params(ng, ngo))
    want = _spectral(rho)
    tol = 2.0**-24 * (1 + 2.0**-10) * np.abs(want) + 1e-12 * np.sqrt((want**2).mean())
    assert np.all(np.abs(grad - want) <= tol)
