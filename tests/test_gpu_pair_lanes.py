"""GPU: the FP64 mode-tile kernels with two lanes per output pair (small solo
grids) against one lane per pair (batches of runs): the same bits.  And the
mixed form's (0,0) mode, whose rows are shared by four lanes, against the FP64
run: its profiles of w and p within the mixed form's 1e-6."""
import numpy as np
import pytest

from f90_dns_gb300 import Batch, ChannelDNS, config_from
from f90_dns_gb300.capi import PREC_MIXED
from f90_dns_gb300.workloads import WORKLOADS

pytestmark = pytest.mark.gpu
C1 = WORKLOADS["channel_32x32x33_re180_dpdx"]
GRIDS = [(16, 12, 6), (16, 12, 7), (32, 24, 17), (32, 32, 34)]


@pytest.mark.parametrize("weak,solver", [(False, 0), (True, 0), (False, 1)])
def test_two_lanes_give_the_bits_of_one(built_lib, weak, solver):
    cfgs = [config_from(dict(C1, nx=a, ny=b, nz=c, use_weak_form_divergence=weak, linear_solver=solver,
                             cgstol=1e-12, perturbation_amplitude=0.05)) for a, b, c in GRIDS]
    solo = []
    for cfg in cfgs:
        with ChannelDNS(cfg) as d:
            d.step(3)
            solo.append(d.get_state())
    runs = [ChannelDNS(cfg) for cfg in cfgs]
    try:
        with Batch(runs) as b:
            b.step(3)
        for r, s in zip(runs, solo):
            st = r.get_state()
            for k in ("u", "v", "w", "p_total"):
                assert np.array_equal(st[k], s[k]), (r.shape, k)
    finally:
        for r in runs:
            r.close()


@pytest.mark.parametrize("nz", [5, 16, 33, 96, 129])
def test_mixed_mean_mode_profile(built_lib, nz):
    wl = dict(C1, nx=16, ny=12, nz=nz, lgl_dmatrix_guard=nz < 58, perturbation_amplitude=0.05)
    prof = []
    for kw in ({}, {"precision": PREC_MIXED}):
        with ChannelDNS(config_from(wl, **kw)) as d:
            d.step(3)
            st = d.get_state()
        prof.append([np.mean(st[k], axis=(1, 2)) for k in ("w", "p_total")])
    for a, b in zip(*prof):
        assert np.max(np.abs(a - b)) <= 1e-6 * max(np.max(np.abs(a)), 1e-3)
