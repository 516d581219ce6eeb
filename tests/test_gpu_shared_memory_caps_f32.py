"""The FP32 evaluation's last admitted sizes, at 48 KB of dynamic shared memory beside its static words, in a
process whose kernels have not been given more before."""
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
nm, nq, nz = 1, 2, 3
mt, mr, rz = (D.as_device(x) for x in (np.array([1e8]) * C.MSOL, np.array([0.1, 1.0]), np.linspace(0.1, 3, nz)))
dens = torch.ones((nm, nq, nz), dtype=torch.float64, device="cuda")
hard = types.SimpleNamespace(_sepa_init=1e3 * C.PC, _num_steps=30, _rchar=100 * C.PC, _gamma_inner=-1.0,
                             _gamma_outer=2.5, _norm_device=lambda: torch.full((nm, nq), 1e7, dtype=torch.float64))


def call(nf):   # phase 2 alone, on one bracketed time an element
    out = [torch.full((nm, nq, nz, nf), v, dtype=torch.float64, device="cuda") for v in (0.0, 5.0 * C.GYR)]
    fobs = np.linspace(1.0, 2.0, nf) / (16 * C.YR)
    rf, dn = sam_cyutils.dbn_2pwl_device(fobs, hard, dens, mt, mr, rz, torch.zeros_like(dens), phase=2, out=out,
                                         precision="fp32")
    torch.cuda.synchronize()
    assert bool((dn > 0.0).all()) and bool((rf > 0.0).all())


top = (48 * 1024 - 40 * ni) // 4
for nf in range(top - 12, top + 1):
    call(nf)
try:
    call(top + 1)
except ValueError:
    print("refused beyond")
"""


def test_sizes_up_to_the_cap(built_lib):
    out = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-2000:]
    assert "refused beyond" in out.stdout
