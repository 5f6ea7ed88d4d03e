"""GPU: the nonlinear term's transforms (fft_nl.cu) over every transform length
they are compiled for.

FP64: the integer chain (inverse y pass, one x kernel with the products, forward
y pass) against the same steps on the FP64-pipe transforms
(DNS3D_FFT_FP64=1: separate c2r, product and r2c kernels), on random fields with
every mode excited: 1e-13 of the velocity scale after 2 steps, the bar the two
transforms are held to over 20 steps of a smooth flow.  Mixed: within the
mixed form's 1e-6 of FP64.  A non-finite value must reach the diagnostics.
"""
import numpy as np
import pytest

from f90_dns_gb300 import ChannelDNS, config_from
from f90_dns_gb300.capi import DNS3D_E_NONFINITE, PREC_MIXED, Dns3DError
from f90_dns_gb300.workloads import WORKLOADS

pytestmark = pytest.mark.gpu

C1 = WORKLOADS["channel_32x32x33_re180_dpdx"]

# every x length nx/2 and every y length ny once, and the ragged ends: rows
# that do not fill the last CTA (nz ny not a multiple of its rows)
GRIDS = [(32, 16, 5), (48, 24, 7), (64, 32, 5), (96, 48, 7), (128, 64, 5), (192, 96, 5), (256, 128, 5),
         (384, 192, 3), (512, 256, 3), (32, 384, 3), (64, 512, 3), (48, 96, 4), (96, 32, 3)]


def _fields(nx, ny, nz, scales=(1.0, 1.0, 1.0)):
    rng = np.random.default_rng(nx * 7 + ny * 3 + nz)
    f = {k: s * rng.standard_normal((nz, ny, nx)) for k, s in zip(("u", "v", "w"), scales)}
    for a in f.values():
        a[0] = a[-1] = 0.0
    f["p_total"] = np.zeros((nz, ny, nx))
    return f


def _run(wl, fields, n, **kw):
    with ChannelDNS(config_from(dict(wl, dt=1e-4), **kw)) as d:
        d.set_state(**fields)
        d.step(n)
        return d.get_state(walls=False)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("dealias", [True, False])
def test_integer_chain_matches_fp64_transforms(built_lib, monkeypatch, grid, dealias):
    nx, ny, nz = grid
    wl = dict(C1, nx=nx, ny=ny, nz=nz, use_dealias_23_rule=dealias)
    f = _fields(nx, ny, nz)
    monkeypatch.setenv("DNS3D_FFT_FP64", "0")
    a = _run(wl, f, 2)
    monkeypatch.setenv("DNS3D_FFT_FP64", "1")
    b = _run(wl, f, 2)
    scale = max(np.max(np.abs(b[k])) for k in ("u", "v", "w"))
    for k in ("u", "v", "w"):
        assert np.max(np.abs(a[k] - b[k])) <= 1e-13 * scale, k


@pytest.mark.parametrize("scales", [(1e6, 1e-6, 1.0), (1e-150, 1e-150, 1e-150), (0.0, 0.0, 1.0)])
def test_integer_chain_over_magnitudes(built_lib, monkeypatch, scales):
    """Rows of very different magnitudes: every product is aligned to the
    larger of its two terms, whatever the fields' own scales."""
    nx, ny, nz = 48, 32, 6
    wl = dict(C1, nx=nx, ny=ny, nz=nz, target_pressure_gradient=0.0)
    f = _fields(nx, ny, nz, scales)
    out = []
    for pipe in ("0", "1"):
        monkeypatch.setenv("DNS3D_FFT_FP64", pipe)
        out.append(_run(wl, f, 1))
    scale = max(np.max(np.abs(out[1][k])) for k in ("u", "v", "w"))
    for k in ("u", "v", "w"):
        assert np.all(np.isfinite(out[0][k]))
        assert np.max(np.abs(out[0][k] - out[1][k])) <= 1e-13 * scale, k


@pytest.mark.parametrize("grid", GRIDS)
def test_mixed_chain_matches_fp64(built_lib, grid):
    nx, ny, nz = grid
    wl = dict(C1, nx=nx, ny=ny, nz=nz)
    f = _fields(nx, ny, nz)
    a = _run(wl, f, 2, precision=PREC_MIXED)
    b = _run(wl, f, 2)
    scale = max(np.max(np.abs(b[k])) for k in ("u", "v", "w"))
    for k in ("u", "v", "w"):
        assert np.max(np.abs(a[k] - b[k])) <= 1e-6 * scale, k


@pytest.mark.parametrize("precision", [0, PREC_MIXED])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_values_reach_the_diagnostics(built_lib, precision, bad):
    nx, ny, nz = 48, 32, 6
    f = _fields(nx, ny, nz)
    f["v"][3, 5, 7] = bad
    with ChannelDNS(config_from(dict(C1, nx=nx, ny=ny, nz=nz), precision=precision)) as d:
        d.set_state(**f)
        d.step(1)
        with pytest.raises(Dns3DError) as e:
            d.diagnostics()
        assert e.value.code == DNS3D_E_NONFINITE
