"""The general two-pass stage (plane pass over 16- and 32-point blocks, stage
pass for any radial block) against the four-kernel stage of the same run,
and that stage of every case against the oracle (the runs of
tests/test_variants.py, test_laplacian.py and test_mixed.py have 16- and
32-point blocks and step in two passes).  Cases: both block lengths in either
direction, tiles left half empty by an odd number of 16-point blocks, radial
blocks of 10 to 64 points, open faces, explicit viscosity, the TVD schemes and
FP32 stage states.

Two steps each.  Only the order in which the density-theta term joins the sums
differs, a rounding; FP64 runs are held to 1e-12 of each field's largest
magnitude (tests/test_fused.py's bar).  An FP32 stage state can round the
other way (2^-24 of a perturbation) where the FP64 value lands on a rounding
boundary: 1e-7 of each field's largest magnitude."""
import numpy as np
import pytest

from css_b200 import problem
from css_b200.context import Simulation
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = {
    "hydro-16x16": dict(dims=(40, 48, 80), decomp=(2, 3, 5)),
    "hydro-16x32": dict(dims=(60, 48, 96), decomp=(3, 3, 3)),
    "hydro-32x16": dict(dims=(24, 64, 80), decomp=(2, 2, 5)),
    "hydro-r10": dict(dims=(20, 32, 48), decomp=(2, 2, 3)),
    "hydro-r64": dict(dims=(128, 64, 96), decomp=(2, 2, 3)),
    "hydro-noslip": dict(dims=(40, 48, 48), decomp=(2, 3, 3), top_stress_free=0, bottom_stress_free=0,
                         theta_stress_free=0, mass_diffusion=0, xi_cs=0.9),
    "mhd-16x16": dict(dims=(40, 48, 80), decomp=(2, 3, 5), magnetic=True),
    "mhd-32x16": dict(dims=(60, 64, 48), decomp=(3, 2, 3), magnetic=True),
    "mhd-16x32": dict(dims=(104, 32, 96), decomp=(2, 2, 3), magnetic=True),
    "mhd-conductor": dict(dims=(40, 48, 48), decomp=(2, 3, 3), magnetic=True, theta_perf_conductor=1,
                          theta_normal_field=0, top_radial_field=0, bottom_radial_field=0, top_perfect_cond=1,
                          bottom_perfect_cond=1),
    "open-both": dict(dims=(64, 64, 96), decomp=(2, 2, 3), top_inout=1, bot_inout=1),
    "open-rain-16": dict(dims=(40, 48, 48), decomp=(2, 3, 3), top_inout=1, do_entropy_rain=1, delta_s=1e-4),
    "viscous-mhd": dict(dims=(64, 64, 96), decomp=(2, 2, 3), magnetic=True, laplacian=1),
    "viscous-16": dict(dims=(40, 48, 48), decomp=(2, 3, 3), laplacian=1),
    "rk2": dict(dims=(40, 48, 48), decomp=(2, 3, 3), time_stepper=2),
    "rk3-32": dict(dims=(64, 64, 96), decomp=(2, 2, 3), time_stepper=3),
    "mixed-32": dict(dims=(64, 64, 96), decomp=(2, 2, 3), precision=1),
    "mixed-16": dict(dims=(40, 48, 80), decomp=(2, 3, 5), precision=1),
    "mixed-mhd-32": dict(dims=(64, 64, 96), decomp=(2, 2, 3), magnetic=True, precision=1),
    "mixed-mhd-16x32": dict(dims=(60, 48, 96), decomp=(3, 3, 3), magnetic=True, precision=1),
    # FP64 slab too large for shared memory, FP32 ones not: stage 1 alone takes the four kernels
    "mixed-mhd-r60": dict(dims=(120, 32, 48), decomp=(2, 2, 3), magnetic=True, precision=1),
    "mixed-rk3": dict(dims=(40, 48, 48), decomp=(2, 3, 3), precision=1, time_stepper=3),
}


@pytest.mark.parametrize("name", list(CASES))
def test_general_stage_equals_four_kernels(name, gpu_available):
    kw = dict(CASES[name])
    p, prof, v0, dt, _ = problem.build(kw.pop("dims"), decomp=kw.pop("decomp"), magnetic=kw.pop("magnetic", False))
    for k, val in kw.items():
        setattr(p, k, val)
    rng = np.random.default_rng(8)
    v0 = v0.copy()
    v0[1:4] = 1e-3 * rng.standard_normal(v0[1:4].shape)
    if p.laplacian:
        dt = 0.1 * dt
    out = []
    for four in (False, True):
        sim = Simulation(p, prof)
        if four:
            sim.set_fused(False)
        sim.upload(v0)
        if p.top_inout or p.bot_inout:
            sim.inout_init()
            sim.set_clock(0, 0.0, dt)
            if p.do_entropy_rain:
                sim.set_rain_fields(*(1e-3 * rng.standard_normal((2, p.nphi, p.nth)) if not out else rain))
            rain = sim.rain_fields()
        n0 = sim.launches()
        sim.step_rk4(dt, 2)
        out.append((sim.download(), sim.launches() - n0))
        sim.close()
    (two, n2), (four_, n4) = out
    assert n2 < n4  # the two forms did run
    bar = 1e-7 if p.precision else 1e-12
    for i in range(two.shape[0]):
        assert np.abs(two[i] - four_[i]).max() <= bar * np.abs(four_[i]).max(), (name, i)


# a prescribed bottom (ASH slices), with 16- and 32-point theta blocks
ASH = {
    "ash-16": dict(dims=(40, 48, 80), decomp=(2, 3, 5), bot_inout=1, bottom_specified=1, ufreq=2),
    "ash-32": dict(dims=(64, 64, 96), decomp=(2, 2, 3), top_inout=1, bot_inout=1, bottom_specified=1, ufreq=2),
}
# the four kernels alone: 24-point theta and phi blocks, which have no two-pass
# stage, with FP32 stage states
FOUR = {
    "mixed-24": dict(dims=(40, 48, 72), decomp=(2, 2, 3), precision=1),
    "mixed-mhd-24": dict(dims=(40, 48, 72), decomp=(2, 2, 3), magnetic=True, precision=1),
}


def case(kw):
    """Parameters, profiles, a stirred state and a time step."""
    kw = dict(kw)
    p, prof, v0, dt, _ = problem.build(kw.pop("dims"), decomp=kw.pop("decomp"), magnetic=kw.pop("magnetic", False))
    for k, val in kw.items():
        setattr(p, k, val)
    v = v0.copy()
    v[1:4] = 1e-3 * np.random.default_rng(8).standard_normal(v[1:4].shape)
    if p.laplacian:
        dt = 0.1 * dt
    return p, prof, v, dt


def open_faces(p, run, v, dt):
    """The open faces' state of a run (device or oracle), from the seeds above."""
    if not (p.top_inout or p.bot_inout):
        return
    rng = np.random.default_rng(9)
    if isinstance(run, Simulation):
        run.inout_init()
    else:
        run.inout_init(v)
    run.set_clock(0, 2.01e5 if p.bottom_specified else 0.0, dt)
    if p.do_entropy_rain:
        sq = np.stack([rng.uniform(p.th1, p.th2, 12), rng.uniform(p.phi1, p.phi2, 12), rng.uniform(0.02, 0.08, 12),
                       np.ones(12), rng.uniform(-2e-3, -1e-3, 12), rng.uniform(-2e-4, -1e-4, 12)], axis=1)
        run.build_squalls(sq)
    if p.bottom_specified:
        run.set_ash_slices(1e-3 * rng.standard_normal((4, 4, p.nphi, p.nth)),
                           np.array([1.9e5, 2.0e5, 2.1e5, 2.2e5]), 1.3)


@pytest.mark.parametrize("name", list(ASH))
def test_prescribed_bottom(name, gpu_available):
    """The general stage under a prescribed bottom: the four kernels to a
    rounding and the oracle to 1e-10, as the runs of tests/test_inout.py."""
    p, prof, v, dt = case(ASH[name])
    out = []
    for four in (False, True):
        sim = Simulation(p, prof)
        assert sim.stage_form == 2
        if four:
            sim.set_fused(False)
        sim.upload(v)
        open_faces(p, sim, v, dt)
        sim.step_rk4(dt, 3)
        out.append(sim.download())
        sim.close()
    orc = O.Oracle(p, prof)
    open_faces(p, orc, v, dt)
    want = orc.step(v, dt, 3)
    for i in range(5):
        assert np.abs(out[0][i] - out[1][i]).max() <= 1e-12 * np.abs(out[1][i]).max(), (name, i)
        assert np.abs(out[0][i] - want[i]).max() <= 1e-10 * np.abs(want[i]).max(), (name, i)


@pytest.mark.parametrize("name", list(CASES) + list(ASH) + list(FOUR))
def test_four_kernels_against_the_oracle(name, gpu_available):
    """Two steps at the bars of the whole runs: FP64 1e-10 of each field's
    largest magnitude (tests/test_gpu_parity.py), FP32 stage states 1e-6 for
    rho and s and 1e-5 for the others (tests/test_mixed.py)."""
    p, prof, v, dt = case({**CASES, **ASH, **FOUR}[name])
    sim, orc = Simulation(p, prof), O.Oracle(p, prof)
    sim.set_fused(False)
    sim.upload(v)
    open_faces(p, sim, v, dt)
    open_faces(p, orc, v, dt)
    sim.step_rk4(dt, 2)
    got, want = sim.download(), orc.step(v, dt, 2)
    sim.close()
    for i in range(got.shape[0]):
        bar = (1e-6 if i in (0, 4) else 1e-5) if p.precision else 1e-10
        assert np.abs(got[i] - want[i]).max() <= bar * np.abs(want[i]).max(), (name, i)


@pytest.mark.parametrize("dims,decomp,form,kw", [
    ((40, 48, 80), (2, 3, 5), 2, {}), ((64, 64, 96), (2, 2, 3), 2, dict(precision=1)),
    ((64, 64, 96), (2, 2, 3), 1, {}), ((40, 48, 72), (2, 2, 3), 0, {})])
def test_form_is_put_back(dims, decomp, form, kw, gpu_available):
    """Switched off and set back to what it was, every run steps in the form it
    had, bit for bit; what a run does not qualify for is refused."""
    from css_b200 import _lib
    from css_b200._lib import CssError
    p, prof, v0, dt, _ = problem.build(dims, decomp=decomp)
    for k, val in kw.items():
        setattr(p, k, val)
    sims = [Simulation(p, prof) for _ in range(2)]
    was = _lib.lib().css_get_fused(sims[1].h)
    assert was == form == sims[1].stage_form and sims[1].fused == (form == 1)
    sims[1].set_fused(False)
    assert sims[1].stage_form == 0 and not sims[1].fused
    if form != 1:
        with pytest.raises(CssError):
            sims[1].set_fused(True)
    if form == 0:
        with pytest.raises(CssError):
            sims[1].set_fused(2)
    else:
        sims[1].set_fused(2)
        assert sims[1].stage_form == form
        sims[1].set_fused(False)
    _lib.check(_lib.lib().css_set_fused(sims[1].h, was))
    assert sims[1].stage_form == form
    for sim in sims:
        sim.upload(v0)
        sim.step_rk4(dt, 2)
    assert np.array_equal(sims[0].download(), sims[1].download())
    assert sims[0].launches() == sims[1].launches()
    for sim in sims:
        sim.close()


def test_no_room_for_the_two_passes(gpu_available):
    """A run that fits the device's memory but for the two passes' own buffer
    is made all the same and steps through the four kernels: as a run switched
    to them, bit for bit."""
    import torch
    p, prof, v0, dt, _ = problem.build((40, 32, 1024), decomp=(2, 2, 32))
    rtw = p.nr * p.nphi * 64 * 8

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    sim = Simulation(p, prof)  # kernels of both forms loaded
    sim.upload(v0)
    sim.step_rk4(dt, 1)
    sim.set_fused(False)
    sim.upload(v0)
    sim.step_rk4(dt, 2)
    want = sim.download()
    with_all = free()
    sim.close()
    need = free() - with_all
    # leave what the run needs less half of that buffer
    hog = torch.empty(free() - need + rtw // 2, dtype=torch.uint8, device="cuda")
    try:
        sim = Simulation(p, prof)
        assert sim.stage_form == 0
        sim.upload(v0)
        sim.step_rk4(dt, 2)
        assert np.array_equal(sim.download(), want)
        sim.close()
    finally:
        del hog
        torch.cuda.empty_cache()


@pytest.mark.parametrize("nr", [44, 100, 200])  # radial blocks of 22, 50 and 100 points
@pytest.mark.parametrize("perfect", [0, 1])
def test_curl_of_any_radial_block(nr, perfect, gpu_available):
    """B of a magnetic run whose radial blocks have a run-time length
    (k_curl_rg: 128, 64 and 32 lines a CTA) against the oracle, both forms of
    the walls' conditions; the FP64 bar of one derivative pass, 1e-12."""
    p, prof, v0, _, _ = problem.build((nr, 28, 66), decomp=(2, 2, 3), magnetic=True)
    p.theta_perf_conductor, p.theta_normal_field = perfect, 1 - perfect
    p.top_radial_field = p.bottom_radial_field = 1 - perfect
    p.top_perfect_cond = p.bottom_perfect_cond = perfect
    v0 = v0.copy()
    v0[5:] = np.random.default_rng(3).standard_normal(v0[5:].shape)
    sim = Simulation(p, prof)
    b = sim.rhs(v0, 1)[0][5:]
    sim.close()
    want = O.Oracle(p, prof).rhs(v0, 1)[0][5:]
    for i in range(3):
        assert np.abs(b[i] - want[i]).max() <= 1e-12 * np.abs(want[i]).max(), i
