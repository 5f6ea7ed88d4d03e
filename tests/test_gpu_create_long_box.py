"""GPU: boxes so long that k^2 vanishes beside the stiffness matrix: the mixed
form refuses what the FP64 form refuses (nz = 3, whose even block has a zero last
pivot then) and accepts what it accepts."""
import pytest

from f90_dns_gb300 import ChannelDNS, Dns3DError, config_from
from f90_dns_gb300.capi import PREC_FP64, PREC_MIXED
from f90_dns_gb300.workloads import WORKLOADS

pytestmark = pytest.mark.gpu
C1 = WORKLOADS["channel_32x32x33_re180_dpdx"]


@pytest.mark.parametrize("box", [dict(xlen=1e10), dict(ylen=1e10), dict(xlen=1e5), {}])
@pytest.mark.parametrize("nz", [3, 4, 5])
def test_mixed_refuses_what_fp64_refuses(built_lib, nz, box):
    codes = []
    for prec in (PREC_FP64, PREC_MIXED):
        try:
            ChannelDNS(config_from(dict(C1, nx=16, ny=16, nz=nz, **box), precision=prec)).close()
            codes.append(0)
        except Dns3DError as e:
            codes.append(e.code)
    assert codes[0] == codes[1]
    assert (codes[0] != 0) == (nz == 3 and 1e10 in box.values())
