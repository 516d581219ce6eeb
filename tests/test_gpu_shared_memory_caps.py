"""The separation-step walk and its evaluation at every size around 48 KB of dynamic shared memory, in a
process whose kernels have not been given more before: the default limit counts static shared memory too."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import types
import numpy as np
import torch
from holodeck_gb300 import _device as D, constants as C
from holodeck_gb300.cosmology import cosmo
from holodeck_gb300.sams import sam_cyutils

ni = int(D.device_cosmology(cosmo).struct.grid_size)
nq, nz = 4, 20
mt, mr, rz = (D.as_device(x) for x in (np.logspace(7, 9, 2) * C.MSOL, np.logspace(-1, 0, nq), np.linspace(0.1, 3, nz)))
gmt = torch.zeros((2, nq, nz), dtype=torch.float64, device="cuda")
dens = torch.ones_like(gmt)


def call(steps, nf):
    hard = types.SimpleNamespace(_sepa_init=1e3 * C.PC, _num_steps=steps, _rchar=100 * C.PC, _gamma_inner=-1.0,
                                 _gamma_outer=2.5, _norm_device=lambda: torch.full((2, nq), 1e7, dtype=torch.float64))
    fobs = np.linspace(1.0, 2.0, nf) / (16 * C.YR)
    rf, dn = sam_cyutils.dbn_2pwl_device(fobs, hard, dens, mt, mr, rz, gmt)
    torch.cuda.synchronize()
    assert bool(torch.isfinite(dn).all())


def walk_bytes(steps, nf, qc):
    return 8 * (3 * ni + nf + nz + 3 * (steps + 1) + nz + qc * (steps + 1)) + 4 * (3 * ni + nf + steps + 1) + 4 * (nf | 1) * nz


n = 0
for steps in range(20, 1500, 5):   # ascending, so a cap raised for one size does not cover the next
    if 44 * 1024 < walk_bytes(steps, 20, 1) < 50 * 1024:
        call(steps, 20)
        n += 1
assert n > 20, n
for nf in range(6144 - 5 * ni - 400, 6144 - 5 * ni + 1, 16):   # the evaluation: 8 (5 ni + nf) up to 48 KB
    if nf > 0:
        call(30, nf)
        n += 1
print("calls", n)
"""


def test_sizes_around_the_default_cap(built_lib):
    out = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-2000:]
