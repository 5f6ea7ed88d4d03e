"""GPU: fields that are constant in x and y come back from set_state and
get_state as they went in, bit for bit, on power-of-two grids up to 128 x 256
points per plane.  The mean mode is then nx ny times the value, every sum of the fixed-point
transforms is exact (a row's or column's one value has 53 bits, which lengths
nx/2 <= 64 and ny <= 256 leave room for), the inverse transforms copy it and
1/(nx ny) is a power of two."""
import numpy as np
import pytest

from f90_dns_gb300 import ChannelDNS, config_from
from f90_dns_gb300.workloads import WORKLOADS

pytestmark = pytest.mark.gpu
C1 = WORKLOADS["channel_32x32x33_re180_dpdx"]


@pytest.mark.parametrize("nx,ny", [(32, 16), (32, 64), (64, 256), (128, 128)])
def test_constant_planes_come_back(built_lib, nx, ny):
    nz = 9
    v = np.random.default_rng(nx + ny).standard_normal((4, nz)) * 10.0 ** np.arange(-4, 5)
    f = np.broadcast_to(v[:, :, None, None], (4, nz, ny, nx)).copy()
    with ChannelDNS(config_from(dict(C1, nx=nx, ny=ny, nz=nz))) as d:
        d.set_state(u=f[0], v=f[1], w=f[2], p_total=f[3])
        st = d.get_state()
    for i, k in enumerate(("u", "v", "w", "p_total")):
        assert np.array_equal(st[k], f[i]), k
