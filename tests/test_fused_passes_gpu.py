"""The strided-axis passes on warp-owned transforms (k_line) and the fused
x forward + RHS + x inverse of RK3 stages 0 and 1 (k_xrhs), at the lengths
where their tiles, masks and box kinds change, against the CPU FP64 oracle.
Tolerances as in test_gpu_parity.py; a few steps of the FP32 form stay
within 1e-6 of the oracle (one RHS of 2e-5 times dt |dU| / |U| < 1e-2 a stage).
"""
import numpy as np
import pytest

import oracle as O
from fields import random_solenoidal, to_spectral
from spooky_b200 import Context, Ensemble
from spooky_b200.initial import masked_noise_state
from spooky_b200.params import SPK_FORM_FP32, SPK_FORM_PLAIN, default_params

pytestmark = pytest.mark.gpu
FORMS = [SPK_FORM_PLAIN, SPK_FORM_FP32]
TOL_STEP = {SPK_FORM_PLAIN: 1e-12, SPK_FORM_FP32: 1e-6}
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


def check_steps(p, U, nsteps, tol):
    o = O.Oracle(p)
    o.set_state(U)
    o.step(nsteps)
    ctx = Context(p)
    ctx.set_state(U)
    ctx.advance(nsteps)
    ctx.synchronize()
    assert rel_l2(ctx.get_state(), o.get_state()) < tol


# every x length k_xrhs covers (24 in the FP32 form only: the plain form runs
# k_axis2 there); 24 y rows and 9 kz columns leave ragged tiles
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("outside", [False, True])
@pytest.mark.parametrize("mhd", [0, 1])
@pytest.mark.parametrize("nx", [24, 32, 48, 64, 96, 128, 192, 256])
def test_fused_stage_matches_oracle(nx, mhd, outside, form):
    p = params((nx, 24, 16), mhd, form)
    check_steps(p, state(p, 5, outside), 3, TOL_STEP[form])


# several k blocks, the last one partial; and no dealiasing (every mode kept)
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("antialiasing", [1, 0])
def test_fused_stage_many_columns(antialiasing, form):
    p = params((64, 16, 96), 1, form, antialiasing=antialiasing)
    check_steps(p, state(p, 6, False), 2, TOL_STEP[form])


# boxes with and without content outside the mask in one group: the fused
# pass takes both kinds of box in one launch
@pytest.mark.parametrize("form", FORMS)
def test_fused_stage_mixed_group(form):
    ps = [params((48, 24, 32), 1, form) for _ in range(3)]
    for p, nu in zip(ps, (1e-2, 5e-3, 2e-3)):
        p.nu = nu
    Us = [state(p, 7 + i, i == 1) for i, p in enumerate(ps)]
    ens = Ensemble(ps)
    for b, U in zip(ens.boxes, Us):
        b.set_state(U)
    ens.advance(3)
    ens.synchronize()
    for p, U, b in zip(ps, Us, ens.boxes):
        o = O.Oracle(p)
        o.set_state(U)
        o.step(3)
        assert rel_l2(b.get_state(), o.get_state()) < TOL_STEP[form]


# every length k_line covers along y (24 in the FP32 form only, 384 in the
# plain form only: k_axis2 runs the other form there), with more than one k block
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


# the same lengths where the y inverse loads the kept rows alone (a prefix and
# a suffix from a multiple of 8) and the x forward filters its outer rows: steps
# from a state inside the mask
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("ny", [24, 32, 48, 64, 96, 128, 192, 256, 384])
def test_trimmed_line_pass_matches_oracle(ny, form):
    p = params((32, ny, 48), 1, form)
    check_steps(p, state(p, 10, False), 2, TOL_STEP[form])


# HD: the odd channel (3 in, 5 out) pairs with itself on the next line of a
# z-pass CTA, in the products and in to_real; from one lane to several warps a
# transform, 48 lines (the last CTA may have fewer)
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("nz", [8, 32, 96, 256, 512, 768, 1024])
def test_odd_channel_pairs_match_oracle(nz, form):
    import torch
    p = params((6, 8, nz), 0, form)
    U = state(p, 12, True)
    ctx = Context(p)
    Ud = torch.from_numpy(U).cuda()
    dU = torch.zeros_like(Ud)
    ctx.compute_dfield(Ud, dU)
    assert rel_l2(dU.cpu().numpy(), O.Oracle(p).compute_dfield(U)) < TOL_RHS[form]
    check_steps(p, U, 2, TOL_STEP[form])
    o = O.Oracle(p)
    o.set_state(U)
    ctx.set_state(U)
    R = torch.zeros(ctx.shape_r, dtype=torch.float64, device="cuda")
    ctx.to_real(R)
    ctx.synchronize()
    assert rel_l2(R.cpu().numpy(), o.to_real()) < (1e-13 if form == SPK_FORM_PLAIN else 1e-6)


# the schedule leaves the values alone: lines per z-pass CTA (HD pairs lines,
# so an odd number is rounded up) and stages of the axis passes
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("shape", [(24, 24, 32), (48, 64, 16), (96, 32, 256), (32, 128, 16), (256, 192, 8)])
def test_schedule_keeps_the_bits(shape, form):
    p = params(shape, 0, form)
    U = state(p, 13, False)

    def run(**knobs):
        ctx = Context(p)
        ctx.set_schedule(**knobs)
        ctx.set_state(U)
        ctx.advance(2)
        ctx.synchronize()
        return ctx.get_state()

    ref = run()
    for knobs in [dict(z_lines=n) for n in (1, 2, 3, 4, 8)] + [dict(axis_stages=n) for n in (1, 2, 3, 4)]:
        assert np.array_equal(run(**knobs), ref), knobs

# the pass table names what a step runs: its launches add up to the step's
# (less k_reset_max, k_dt and k_masked_rk) within the seven entries a caller
# provides, and the kernels it times are the step's.  nx = 16 has no fused pass.
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("nx", [16, 32])
def test_profiled_passes_are_those_of_a_step(nx, form):
    import ctypes
    from torch.profiler import ProfilerActivity, profile
    from spooky_b200 import PassStat, lib
    p = params((nx, 32, 32), 1, form)
    ctx = Context(p)
    ctx.set_state(state(p, 11, False))
    ctx.advance(2)
    ctx.synchronize()
    out, n = (PassStat * 7)(), ctypes.c_int()

    def kernels(call):
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            call()
            ctx.synchronize()
        return {e.name for e in prof.events() if "spk::" in e.name}

    steps = kernels(lambda: ctx.advance(2))
    timed = kernels(lambda: ctx._check(lib().spk_profile_passes(ctx._h, 1, out, 7, ctypes.byref(n))))
    assert steps and timed and timed <= steps, timed - steps
    table = {out[i].name.decode(): out[i].launches_per_step for i in range(n.value)}
    assert sum(table.values()) == ctx.step_info()[0] - 3
    assert ("x_fwd_rhs_x_inv" in table) == (nx == 32) and 0 not in table.values()
