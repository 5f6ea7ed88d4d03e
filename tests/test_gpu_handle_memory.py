"""GPU: a handle holds the device memory of what it builds.  At 128x96x129 the
tensor-core images (digit slices of the Helmholtz inverses, fixed-point Poisson
inverses) are half of an FP64 handle; with DNS3D_TENSOR_CORES=0 none is built
and none is held.  Sizes from the operators: nq = 65 x 49 wavenumber pairs, a
fixed-point inverse of 65^2 + 64^2 (+1) 64-bit integers each; the driver hands
out memory in 2 MB pages, the library adds at most a block of 4 MB."""
import pytest

from f90_dns_gb300 import ChannelDNS, config_from, footprint_bytes
from f90_dns_gb300.workloads import WORKLOADS

pytestmark = pytest.mark.gpu
C1 = WORKLOADS["channel_32x32x33_re180_dpdx"]


def _held(torch, cfg):
    free = torch.cuda.mem_get_info()[0]
    with ChannelDNS(cfg):
        return free - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("precision", [0, 1])
def test_memory_held(built_lib, monkeypatch, precision):
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda")
    cfg = config_from(dict(C1, nx=128, ny=96, nz=129, lgl_dmatrix_guard=False), precision=precision)
    monkeypatch.setenv("DNS3D_AUTOTUNE", "0")
    _held(torch, cfg)  # modules loaded, contexts and pools grown
    on = _held(torch, cfg)
    monkeypatch.setenv("DNS3D_TENSOR_CORES", "0")
    off = _held(torch, cfg)
    poisson = 65 * 49 * (65 * 65 + 64 * 64 + 1) * 8
    mb = 1 << 20
    assert on <= footprint_bytes(cfg) + 8 * mb
    if precision == 0:
        assert off <= on - poisson
    else:
        assert abs(on - off) <= 4 * mb
