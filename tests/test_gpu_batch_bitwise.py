"""GPU: runs that a batch takes into its shared launches (every length with
compile-time transforms, checked by the batch's own count) equal their solo
runs bitwise.  Small solo runs take two lanes per output pair in the FP64
vorticity, pressure and projection kernels, batches one; with the tensor cores
forced on, the fixed-point Poisson solve of a batch has 256 threads for the
solo kernel's 64 to 288, with operators per CTA from one (nz = 129) to many."""
import numpy as np
import pytest

from f90_dns_gb300 import Batch, ChannelDNS, config_from
from f90_dns_gb300.capi import PREC_FP64, PREC_MIXED
from f90_dns_gb300.workloads import WORKLOADS

pytestmark = pytest.mark.gpu
C1 = WORKLOADS["channel_32x32x33_re180_dpdx"]
# below the line of two lanes (34048 output pairs) but for the last
GRIDS = [(32, 16, 3), (32, 24, 4), (48, 16, 17), (32, 32, 34), (32, 16, 65), (48, 24, 96), (32, 16, 129), (64, 48, 49)]


def _solo_and_batch(cfgs, steps):
    solo = []
    for cfg in cfgs:
        with ChannelDNS(cfg) as d:
            d.step(steps)
            solo.append(d.get_state())
    runs = [ChannelDNS(cfg) for cfg in cfgs]
    try:
        with Batch(runs) as b:
            assert b.info()[1] == len(runs)  # none stepped by its own launches
            b.step(steps)
        for r, s in zip(runs, solo):
            st = r.get_state()
            for k in ("u", "v", "w", "p_total"):
                assert np.array_equal(st[k], s[k]), (r.shape, k)
    finally:
        for r in runs:
            r.close()


def _cfgs(precision, **kw):
    return [config_from(dict(C1, nx=a, ny=b, nz=c, lgl_dmatrix_guard=c < 58, perturbation_amplitude=0.05, **kw),
                        precision=precision) for a, b, c in GRIDS]


@pytest.mark.parametrize("weak", [False, True])
@pytest.mark.parametrize("precision,tensor_cores", [(PREC_FP64, "0"), (PREC_FP64, "1"), (PREC_MIXED, "0")])
def test_batch_equals_solo(built_lib, monkeypatch, precision, tensor_cores, weak):
    monkeypatch.setenv("DNS3D_TENSOR_CORES", tensor_cores)
    _solo_and_batch(_cfgs(precision, use_weak_form_divergence=weak), 3)


def test_batch_equals_solo_fp64_pipe_transforms(built_lib, monkeypatch):
    monkeypatch.setenv("DNS3D_FFT_FP64", "1")
    _solo_and_batch(_cfgs(PREC_FP64), 2)
