"""GPU: the nonlinear term's y passes with the small tiles of grids that leave
SMs without a CTA (solo runs) against the full tiles (batches): the same bits,
for every length with a remainder of columns."""
import numpy as np
import pytest

from f90_dns_gb300 import Batch, ChannelDNS, config_from
from f90_dns_gb300.workloads import WORKLOADS

pytestmark = pytest.mark.gpu
C1 = WORKLOADS["channel_32x32x33_re180_dpdx"]


@pytest.mark.parametrize("dealias", [True, False])
@pytest.mark.parametrize("ny", [16, 24, 32, 48, 64, 96, 128, 192, 256])
def test_small_tiles_give_the_bits_of_full_ones(built_lib, ny, dealias):
    cfg = config_from(dict(C1, nx=32, ny=ny, nz=5, use_dealias_23_rule=dealias, perturbation_amplitude=0.05))
    with ChannelDNS(cfg) as d:
        d.step(2)
        solo = d.get_state()
    with ChannelDNS(cfg) as r:
        with Batch([r]) as b:
            b.step(2)
        st = r.get_state()
    for k in ("u", "v", "w", "p_total"):
        assert np.array_equal(st[k], solo[k]), k
