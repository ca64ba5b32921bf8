"""Requests that follow one another on a context, and shares of a request, on the GPU."""
import numpy as np
import pytest

from oscars_b200.sr import sr
from cases import BEAM_GAUSS, E1_U, UND_SHORT, run_case, traj

pytestmark = pytest.mark.gpu


def _machine():
    s = sr(gpu=1)
    run_case(s, [UND_SHORT, BEAM_GAUSS] + traj(5001, -0.5, 0.5))
    return s


# A refused request leaves nothing behind: what follows is what a fresh context gives.  (Variants tuned per context
# and FP64 sums in another order: 1e-12 of the peak.)
@pytest.mark.parametrize("side", [2, 100])  # results through mapped memory, and downloads through page-locked memory
@pytest.mark.parametrize("nparticles", [0, 3])
def test_requests_after_a_refused_one(side, nparticles):
    common = dict(max_level=6, nparticles=nparticles, return_numpy=True)
    geo = dict(npoints=[side, side], width=[0.002, 0.002], translation=[0, 0, 20])
    results = []
    for refused in (False, True):
        s = _machine()
        for call in (lambda: s.calculate_flux_rectangle(energy_eV=E1_U, **geo, **common),
                     lambda: s.calculate_spectrum(obs=[0, 0, 20], energy_range_eV=[400, 500], npoints=side * side, **common),
                     lambda: s.calculate_power_density_rectangle(**geo, **common)):
            s.set_new_particle(particle="ideal")
            if refused:
                with pytest.raises(ValueError, match="compute='mixed' needs observers near the beam axis"):
                    s.calculate_flux_rectangle(energy_eV=E1_U, npoints=[side, side], width=[1e-4, 1e-4],
                                               translation=[3, 0, 20], max_level=6, compute="mixed")
            s.set_seed(3)
            results.append(call() + (s.last_levels,))
    for want, got in zip(results[:3], results[3:]):
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[2], want[2])
        assert want[1].min() > 0 and np.max(np.abs(got[1] - want[1])) <= 1e-12 * np.max(want[1])


# A process without a particle of a shared request: the positions of the whole request, zeros, no level.
@pytest.mark.parametrize("compute", ["fp64", "mixed"])
@pytest.mark.parametrize("form", ["rectangle", "three points", "power density"])
def test_share_without_a_particle(compute, form):
    s = _machine()
    geo = dict(npoints=[91, 93], translation=[0.001, 0.002, 20], nparticles=3, max_level=4, compute=compute, return_numpy=True)
    if form == "three points":
        geo["x0x1x2"] = [[-0.001, -0.001, 0], [0.001, -0.001, 0], [-0.001, 0.001, 0]]
    else:
        geo["width"] = [0.002, 0.002]

    def call(**kw):
        s.set_seed(5)
        if form == "power density":
            return s.calculate_power_density_rectangle(**geo, **kw) + (s.last_levels,)
        return s.calculate_flux_rectangle(energy_eV=E1_U, **geo, **kw) + (s.last_levels,)
    pos, values, levels = call(shard=(3, 4))
    whole = call()
    assert np.array_equal(pos, whole[0]) and not values.any() and np.all(levels == -1) and whole[1].min() > 0


# The deepest levels of a few entries fill the chip: at most twice the time that their share of many entries takes
# (1.3 at one tile's 32 observers; 3.1 and 3.6 while a level went in 64 spans whatever its length).
@pytest.mark.parametrize("compute", ["fp64", "mixed"])
def test_deep_levels_of_few_entries_fill_the_chip(compute):
    import time
    s = _machine()

    def seconds(n):
        kw = dict(energy_eV=E1_U, npoints=[n, 1], width=[0.002, 0.002], translation=[0, 0, 20], precision=0.0, max_level=24,
                  compute=compute, return_numpy=True)
        best = np.inf
        for _ in range(4):  # (the first fills the level cache and tunes)
            t = time.perf_counter()
            s.calculate_flux_rectangle(**kw)
            best = min(best, time.perf_counter() - t)
        return best
    assert seconds(32) <= 2.0 * seconds(47 * 32) / 47


# A batch whose jobs all go in energy tiles leaves no choice of the other jobs' kernel behind: a later one with the
# same numbers of jobs and entries, but few energies a job, times its variants as on a fresh context (at 900 entries
# a job another one than a context starts with).
def test_batch_variant_is_timed_for_jobs_of_few_energies():
    from oscars_b200.batch import BatchRunner, Job, undulator

    def jobs(m, n):
        return [Job(fields=[undulator([0, 0.5, 0], [0, 0, 0.05], 11, phase=-np.pi / 2)], energy_GeV=3.0, ctstartstop=(-0.5, 0.5),
                    npoints=5001, obs=[[1e-5 * k, 2e-6 * k, 20.0] for k in range(m)], energies_eV=np.linspace(300, 600, n))] * 2
    fresh, after = BatchRunner(gpu=0), BatchRunner(gpu=0)
    fresh.flux(jobs(100, 9))
    after.flux(jobs(90, 10))
    after.flux(jobs(100, 9))
    assert after.variant() == fresh.variant()


# A beam's last trajectory, made from half trajectories of several threads in kept buffers, is the one of the same
# particle alone, bit for bit: also an RKAS one, whose sums are NaN (its spline holds the start time twice) and so
# show nothing.
@pytest.mark.parametrize("method", ["RK4", "RKAS"])
def test_last_trajectory_of_a_beam(method):
    s = _machine()
    s.set_trajectory_calculation(method, **({} if method == "RK4" else {"precision": 1e-7}))
    for n, points in ((1, 801), (44, 1201), (3, 401)):
        s.set_npoints_trajectory(points)
        s.set_seed(7)
        s.calculate_flux_rectangle(energy_eV=E1_U, npoints=[1, 1], width=[0.002, 0.002], translation=[0, 0, 20], max_level=3,
                                   nparticles=n)
        got = s.trajectory_array().copy()
        s.set_seed(7)
        for _ in range(n):
            s.set_new_particle()
        s.calculate_trajectory()
        want = s.trajectory_array()
        assert np.isfinite(want).all() and np.array_equal(got, want)


# The batch's splines by the rule on its shape, on both sides of its two lines (1000 times the longest trajectory's
# points, 722 times from 8000 points on), are one of the two kernels' splines bit for bit, the one that the rule
# states.
@pytest.mark.parametrize("jobs, npoints, kernel", [(990, 1001, 2), (1010, 1001, 1), (715, 8001, 2), (730, 8001, 1), (3, 8001, 2)])
def test_spline_kernel_by_the_chunks_shape(jobs, npoints, kernel):
    from oscars_b200.batch import BatchRunner, Job, undulator
    job = Job(fields=[undulator([0.1, 0.5, 0], [0, 0, 0.05], 12, phase=-0.7)], energy_GeV=3.0, ctstartstop=(-0.4, 0.5),
              npoints=npoints, obs=[[0, 0, 20]], energies_eV=[400.0])
    got = []
    for mode in (0, 1, 2):
        r = BatchRunner(gpu=0)
        r.ctx.call("osc_set_batch_spline_kernel", mode)
        got.append(r.trajectories([job] * jobs)[-1])
    assert not np.array_equal(got[1], got[2]) and np.array_equal(got[0], got[kernel])
