"""GPU: the fixed-point Poisson solve, whose CTAs take operators with both their
modes (kx, +-ky): heights and mode counts with every remainder of operators per
CTA, ky = 0 and ny/2 (one mode each), the pinned mode beside others.  Bars: the
tensor-core forms' agreement with the FP64 pipe, 1e-13 of
the velocity scale over 3 steps (the pressure: 1e-11 of its own largest value,
whose solve amplifies the right-hand side's rounding by the operator's
condition); batches equal solo runs bitwise."""
import numpy as np
import pytest

from f90_dns_gb300 import Batch, ChannelDNS, config_from
from f90_dns_gb300.workloads import WORKLOADS

pytestmark = pytest.mark.gpu
C1 = WORKLOADS["channel_32x32x33_re180_dpdx"]
GRIDS = [(16, 12, 4), (16, 12, 5), (24, 16, 18), (16, 24, 33), (48, 16, 34), (16, 16, 65), (16, 12, 96), (16, 12, 129)]


def _cfg(nx, ny, nz):
    return config_from(dict(C1, nx=nx, ny=ny, nz=nz, lgl_dmatrix_guard=nz < 58, perturbation_amplitude=0.05))


@pytest.mark.parametrize("nx,ny,nz", GRIDS)
def test_solve_agrees_with_fp64_pipe(built_lib, monkeypatch, nx, ny, nz):
    out = {}
    for tc in ("0", "1"):
        monkeypatch.setenv("DNS3D_TENSOR_CORES", tc)
        with ChannelDNS(_cfg(nx, ny, nz)) as d:
            d.step(3)
            out[tc] = d.get_state()
    scale = max(np.max(np.abs(out["0"][k])) for k in ("u", "v", "w"))
    for k in ("u", "v", "w"):
        assert np.max(np.abs(out["1"][k] - out["0"][k])) <= 1e-13 * scale, k
    assert np.max(np.abs(out["1"]["p_total"] - out["0"]["p_total"])) <= 1e-11 * np.max(np.abs(out["0"]["p_total"]))


def test_batches_bitwise(built_lib, monkeypatch):
    monkeypatch.setenv("DNS3D_TENSOR_CORES", "1")
    cfgs = [_cfg(*g) for g in GRIDS]
    solo = []
    for cfg in cfgs:
        with ChannelDNS(cfg) as d:
            d.step(2)
            solo.append(d.get_state())
    runs = [ChannelDNS(cfg) for cfg in cfgs]
    try:
        with Batch(runs) as b:
            b.step(2)
        for r, s in zip(runs, solo):
            st = r.get_state()
            for k in ("u", "v", "w", "p_total"):
                assert np.array_equal(st[k], s[k]), (r.shape, k)
    finally:
        for r in runs:
            r.close()
