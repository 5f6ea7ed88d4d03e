"""GPU: creating handles.  The mixed form builds the (0,0) mode's inverses only;
it must refuse what the FP64 form, which builds all of them, refuses: a
guarded derivative matrix that is singular and a k^2 that overflows.  Many
handles of different sizes live at once, each in its own memory."""
import numpy as np
import pytest

from f90_dns_gb300 import ChannelDNS, Dns3DError, config_from
from f90_dns_gb300.capi import PREC_FP64, PREC_MIXED
from f90_dns_gb300.workloads import WORKLOADS

pytestmark = pytest.mark.gpu
C1 = WORKLOADS["channel_32x32x33_re180_dpdx"]


@pytest.mark.parametrize("kw", [dict(nx=16, ny=12, nz=65, lgl_dmatrix_guard=True), dict(nx=16, ny=12, nz=17, xlen=1e-200),
                                dict(nx=16, ny=12, nz=17, ylen=1e-200)])
def test_mixed_refuses_what_fp64_refuses(built_lib, kw):
    codes = []
    for prec in (PREC_FP64, PREC_MIXED):
        try:
            ChannelDNS(config_from(dict(C1, **kw), precision=prec)).close()
            codes.append(0)
        except Dns3DError as e:
            codes.append(e.code)
    assert codes[0] == codes[1]
    assert codes[0] != 0 or kw["nz"] != 65


@pytest.mark.parametrize("jst4", [0, 1])
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_handles_side_by_side_equal_handles_alone(built_lib, prec, jst4):
    grids = [(4, 4, 3), (16, 12, 6), (32, 24, 17), (8, 6, 9), (48, 64, 33)]  # 4 x 4, 8 x 6: no compile-time transforms
    cfgs = [config_from(dict(C1, nx=a, ny=b, nz=c, perturbation_amplitude=0.05, convection_scheme=jst4), precision=prec)
            for a, b, c in grids]
    alone = []
    for cfg in cfgs:
        with ChannelDNS(cfg) as d:
            d.step(2)
            alone.append(d.get_state())
    runs = [ChannelDNS(cfg) for cfg in cfgs]
    try:
        for _ in range(2):
            for r in runs:
                r.step(1)
        for r, s in zip(runs, alone):
            st = r.get_state()
            for k in ("u", "v", "w", "p_total"):
                assert np.array_equal(st[k], s[k]), (r.shape, k)
    finally:
        for r in runs:
            r.close()
