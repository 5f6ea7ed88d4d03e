"""GPU: the mixed projection's strong-form right-hand side in double-float
(pressure_mixed_body, df_dot) at odd and even, the smallest and larger heights
and at mode counts that leave a ragged last tile, against the FP64 oracle: the
mixed form's velocity bar of 1e-6 after 5 steps, and its agreement with the
weak form's kernel branch (FP64 combination) on the same bar."""
import numpy as np
import pytest

from f90_dns_gb300 import ChannelDNS, config_from
from f90_dns_gb300.capi import PREC_MIXED
from f90_dns_gb300.workloads import WORKLOADS
from oracle import dns3d_ref as ref
from tests.helpers import oracle_config, scaled_velocity_errors

pytestmark = pytest.mark.gpu
C1 = WORKLOADS["channel_32x32x33_re180_dpdx"]


@pytest.mark.parametrize("weak", [False, True])
@pytest.mark.parametrize("nx,ny,nz", [(16, 24, 5), (16, 24, 6), (24, 16, 34), (16, 24, 65), (16, 16, 97)])
def test_right_hand_side_forms(built_lib, nx, ny, nz, weak):
    wl = dict(C1, nx=nx, ny=ny, nz=nz, lgl_dmatrix_guard=nz < 58, use_weak_form_divergence=weak,
              perturbation_amplitude=0.05)
    with ChannelDNS(config_from(wl, precision=PREC_MIXED)) as d:
        d.step(5)
        st = d.get_state()
    cfg = oracle_config(wl)
    _, ost, _ = ref.run(cfg, 5, record_every=5)
    err = scaled_velocity_errors(st, ost)
    assert max(err["u"], err["v"], err["w"]) <= 1e-6, err
    assert np.all(np.isfinite(st["p_total"]))
