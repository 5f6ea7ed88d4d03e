"""GPU: the mixed projection's right-hand side is formed from the full FP64 u*,
v*, w*.  The divergence of u* is dt times a source, so from a solenoidal state
it is dt of its own terms: a right-hand side that loses bits of the terms
(float pairs hold 2^-48 of them) shows in the residual of the solve as dt gets
small.  The solve itself, in FP32, is linear in its right-hand side: its relative
residual does not depend on dt.  Bar: a factor 3 between dt = 1e-3 and 1e-8, for
the different shapes of the two right-hand sides (D1.w* in double-float with
FP64 combination adds 2e-13 to 2e-12 of the larger one's maximum, nz = 17 to 129, which at
1e-8 is 1e5 times that: below a twentieth of the residuals, 5e-7 to 3e-4)."""
import math

import numpy as np
import pytest

from f90_dns_gb300 import ChannelDNS, config_from
from f90_dns_gb300.capi import PREC_MIXED, lgl_nodes_weights
from f90_dns_gb300.workloads import WORKLOADS

pytestmark = pytest.mark.gpu
C1 = WORKLOADS["channel_32x32x33_re180_dpdx"]


def _solenoidal(nx, ny, z, xlen, ylen):
    """1 - z^2 and the curl of a vector potential, polynomial in z: solenoidal
    on the LGL points too."""
    r = np.random.default_rng(0)
    x, y = np.arange(nx) * (xlen / nx), np.arange(ny) * (ylen / ny)
    f = np.zeros((3, len(z), ny, nx))
    f[0] += (1 - z * z)[:, None, None]
    for _ in range(12):
        kx = int(r.integers(0, nx // 6)) * 2 * math.pi / xlen
        ky = int(r.integers(-(ny // 6), ny // 6 + 1)) * 2 * math.pi / ylen
        a, b, ph = 0.05 * r.standard_normal(3), r.uniform(-1, 1), r.uniform(0, 2 * math.pi)
        g = (1 - z * z) ** 2 * (1 + b * z)
        dg = -4 * z * (1 - z * z) * (1 + b * z) + (1 - z * z) ** 2 * b
        arg = kx * x[None] + ky * y[:, None] + ph
        for c, p, q in ((0, -a[1], -ky * a[2]), (1, a[0], kx * a[2]), (2, 0.0, -kx * a[1] + ky * a[0])):
            f[c] += (p * dg)[:, None, None] * np.cos(arg) + (q * g)[:, None, None] * np.sin(arg)
    return f


@pytest.mark.parametrize("nz", [17, 33, 34, 65, 129])
def test_residual_does_not_grow_as_dt_shrinks(built_lib, nz):
    nx, ny = 32, 24
    f = _solenoidal(nx, ny, np.asarray(lgl_nodes_weights(nz)[0]), C1["xlen"], C1["ylen"])
    res = []
    for dt in (1e-3, 1e-8):
        cfg = config_from(dict(C1, nx=nx, ny=ny, nz=nz, dt=dt, lgl_dmatrix_guard=False), precision=PREC_MIXED)
        with ChannelDNS(cfg) as d:
            d.set_state(u=f[0], v=f[1], w=f[2], p_total=np.zeros_like(f[0]))
            d.step(1)
            res.append(d.projection_residual())
    assert res[1] <= 3 * res[0], res
