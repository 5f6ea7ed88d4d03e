"""GPU: the first handle of a process runs the same kernels as the next ones
(kernel attributes are raised before anything is chosen by them): in a process
of its own, with the tensor cores forced on, both step through the
tensor-core kernels."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
from f90_dns_gb300 import ChannelDNS, config_from
from f90_dns_gb300.workloads import WORKLOADS
cfg = config_from(dict(WORKLOADS["channel_32x32x33_re180_dpdx"], nx=32, ny=32, nz={nz}, lgl_dmatrix_guard=False))
for _ in range(2):
    with ChannelDNS(cfg) as d:
        print(" ".join(sorted(d.profile_kernels(1))))
"""


@pytest.mark.parametrize("nz", [33, 129])
def test_first_handle_has_the_tensor_core_kernels(built_lib, nz):
    env = dict(os.environ, DNS3D_TENSOR_CORES="1", PYTHONPATH=ROOT)
    out = subprocess.run([sys.executable, "-c", CODE.format(nz=nz)], env=env, cwd=ROOT, capture_output=True, text=True,
                         timeout=300, check=True).stdout.split("\n")
    assert out[0] == out[1]
    for k in ("viscous_helmholtz_tc", "vorticity_tc", "pressure_poisson_tc", "pressure_correction_tc"):
        assert k in out[0], out[0]
