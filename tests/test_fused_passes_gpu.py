"""The strided-axis passes on warp-owned transforms (k_line), at the
lengths where its tiles and masks change, against the CPU FP64 oracle.
Tolerances as in test_gpu_parity.py.
"""
import numpy as np
import pytest

import oracle as O
from fields import random_solenoidal, to_spectral
from spooky_b200 import Context
from spooky_b200.initial import masked_noise_state
from spooky_b200.params import SPK_FORM_FP32, SPK_FORM_PLAIN, default_params

pytestmark = pytest.mark.gpu
FORMS = [SPK_FORM_PLAIN, SPK_FORM_FP32]
TOL_RHS = {SPK_FORM_PLAIN: 1e-12, SPK_FORM_FP32: 2e-5}


def rel_l2(a, b):
    return float(np.linalg.norm((a - b).ravel()) / max(np.linalg.norm(b.ravel()), 1e-300))


def params(shape, mhd, form, **kw):
    return default_params(incompressible=1, mhd=mhd, gridsize=shape, boxsize=(1.0, 1.5, 2.0), reynolds=200.0,
                          reynolds_magnetic=100.0, form=form, t_final=1e9, toutput_flow=1e9, **kw)


def state(p, seed, outside):
    """Solenoidal fields inside the 2/3 mask, or with content outside it too."""
    u = list(random_solenoidal(p, seed, kpeak=3.0))
    if p.mhd:
        B = random_solenoidal(p, seed + 50, kpeak=3.0, rms=0.6)
        B[0] += 0.3
        u += list(B)
    U = to_spectral(np.stack(u))
    if p.antialiasing:
        U = U * O.Oracle(p).kgrid()[1]
    return masked_noise_state(p, U, rel=0.2, seed=seed) if outside else U


# every length k_line covers along y, with more than one k block
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("ny", [24, 32, 48, 64, 96, 128, 192, 256, 384])
def test_line_pass_matches_oracle(ny, form):
    import torch
    p = params((16, ny, 48), 1, form)
    U = state(p, 9, True)
    ctx = Context(p)
    Ud = torch.from_numpy(U).cuda()
    dU = torch.zeros_like(Ud)
    ctx.compute_dfield(Ud, dU)
    assert rel_l2(dU.cpu().numpy(), O.Oracle(p).compute_dfield(U)) < TOL_RHS[form]

