"""Sample-sum kernels at the edges of their tiles, spans and branches, against the CPU oracle."""
import numpy as np
import pytest

from oracle.oracle import OracleSR
from oscars_b200.sr import sr
from cases import E1_U, UND_SHORT_SETUP, run_case

pytestmark = pytest.mark.gpu


def _run(o, calls):
    return np.array([r[1] for r in run_case(o, UND_SHORT_SETUP + calls)], dtype=np.float64)


def _both(call, kw):
    return _run(sr(gpu=1), [(call, kw)]), _run(OracleSR(), [(call, kw)])


# Phases, distances and 1 - n.b have the oracle's bits; what differs is an amplitude's last bits (about
# 20 roundings, 4e-15) and sine and cosine (2e-16), so a sum is off by 5e-15 of the sum of its terms'
# magnitudes, which exceeds the map's peak by less than 2000: 1e-11.
@pytest.mark.parametrize("nx, ny, level", [(1, 1, 0), (1, 1, 1), (31, 1, 2), (1, 33, 4), (5, 13, 6), (3, 43, 9), (16, 8, 12)])
def test_fp64_flux_tiles_and_levels(nx, ny, level):
    kw = dict(energy_eV=E1_U, npoints=[nx, ny], width=[0.004, 0.006], translation=[0, 0, 20], max_level=level)
    got, want = _both("calculate_flux_rectangle", kw)
    assert np.max(np.abs(got - want)) <= 1e-11 * np.max(np.abs(want))


# Above 2^49 rad (1e8 eV at 20 m is 1e16) the phases take the library's sine and cosine.
def test_fp64_flux_beyond_the_fast_phases():
    kw = dict(energy_eV=1e8, npoints=[3, 3], width=[0.004, 0.006], translation=[0, 0, 20], max_level=5)
    got, want = _both("calculate_flux_rectangle", kw)
    assert np.max(np.abs(got - want)) <= 1e-9 * np.max(np.abs(want))


# The line kernels (one observer): tiles of 64 energies, spans of 64 samples, and the step test of the
# stop rule at its precise bound (level 9 and up); the same roundings as above.
@pytest.mark.parametrize("n, level", [(1, 0), (2, 3), (63, 8), (64, 9), (65, 10), (129, 12), (40, 13)])
def test_fp64_spectrum_tiles_and_levels(n, level):
    kw = dict(obs=[0.001, 0, 20], energy_range_eV=[200, 1900], npoints=n, max_level=level)
    got, want = _both("calculate_spectrum", kw)
    assert np.max(np.abs(got - want)) <= 1e-11 * np.max(np.abs(want))


# Mixed: every phase, amplitude, sine, cosine and FP32 partial sum is the general kernel's; the order of
# at most 2^9 FP64 additions differs (2^9 x 2^-53 of the sum of magnitudes, < 2000 peaks): 1e-10.
@pytest.mark.parametrize("n, level", [(1, 9), (64, 10), (65, 11), (200, 14)])
def test_mixed_spectrum_lines_match_general_kernel(n, level):
    out = []
    for variant in (0, -1):
        s = sr(gpu=1)
        s._ctx.call("osc_set_variant", 2, variant)
        run_case(s, UND_SHORT_SETUP)
        e, f = s.calculate_spectrum(obs=[0.001, 0, 20], energy_range_eV=[200, 1900], npoints=n, max_level=level,
                                    compute="mixed", return_numpy=True)
        out.append((f, s.last_levels.copy()))
    assert np.array_equal(out[0][1], out[1][1])
    assert np.max(np.abs(out[0][0] - out[1][0])) <= 1e-10 * np.max(np.abs(out[0][0]))


# Power density: N1, N1 . normal and 1 - b.N1 have the oracle's bits, the rest of a term about 40 roundings
# (5e-15), and the terms of a point have one sign: 1e-12.
@pytest.mark.parametrize("nx, ny, normal, plane, level", [(1, 1, 0, "XY", 0), (31, 1, 1, "XY", 3), (3, 11, -1, "XY", 9),
                                                          (5, 13, 0, "XY", 10), (9, 7, 1, "XZ", 11), (8, 16, -1, "YZ", 12)])
def test_fp64_power_density_tiles_and_levels(nx, ny, normal, plane, level):
    kw = dict(npoints=[nx, ny], plane=plane, width=[0.02, 0.03], normal=normal, translation=[0, 0.01, 20], max_level=level)
    got, want = _both("calculate_power_density_rectangle", kw)
    assert np.max(np.abs(got - want)) <= 1e-12 * max(np.max(np.abs(want)), 1e-300)


# A rectangle formed on the device against the same points uploaded: small (staged inputs, results stored by the
# report kernel up to 8192 entries) and larger ones (downloads through page-locked memory).  Same bits.
@pytest.mark.parametrize("nx, ny", [(1, 1), (7, 5), (64, 128), (91, 91)])
@pytest.mark.parametrize("power", [False, True])
def test_rectangle_formed_on_device_matches_uploaded_points(nx, ny, power):
    import ctypes
    from oscars_b200._lib import dptr, i32ptr
    s = sr(gpu=1)
    run_case(s, UND_SHORT_SETUP)
    geo = dict(npoints=[nx, ny], plane="ZY", width=[0.02, 0.03], rotations=[0.1, 1.4, -0.2], translation=[0.001, 0, 20])
    common = dict(geo, dim=3, max_level=9, normal=1, return_numpy=True)
    if power:
        pos, got = s.calculate_power_density_rectangle(**common)
    else:
        pos, got = s.calculate_flux_rectangle(energy_eV=E1_U, **common)
    levels = s.last_levels
    xyz, nrm, _ = s._rectangle(geo["npoints"], geo["plane"], geo["width"], None, geo["rotations"], geo["translation"], 1, power)
    want, lv, nnc = np.zeros(nx * ny), np.zeros(nx * ny, np.int32), ctypes.c_longlong()
    o = s._opts("", 112188979912321.0, None, None, 0.01, 9, 0, 0, 0, "fp64")
    if power:
        s._ctx.call("osc_power_density", dptr(xyz), dptr(nrm), nx * ny, 1, ctypes.byref(o), dptr(want), i32ptr(lv), ctypes.byref(nnc))
    else:
        s._ctx.call("osc_flux", dptr(xyz), nx * ny, E1_U, ctypes.byref(o), dptr(want), i32ptr(lv), ctypes.byref(nnc))
    assert np.array_equal(pos.ravel(), xyz) and np.array_equal(got, want) and np.array_equal(levels, lv)


# Results beyond the page-locked download buffer (64 MiB: 5.6 million entries) go straight into the caller's arrays,
# which the rectangle call clears while the device computes; page-locked arrays take that way at any size.  Same bits.
@pytest.mark.parametrize("nx, ny, locked", [(2400, 2400, False), (91, 91, True)])
def test_rectangle_downloads_straight_into_the_callers_arrays(nx, ny, locked):
    import ctypes
    import torch
    from oscars_b200._lib import dptr, i32ptr, lib
    s = sr(gpu=1)
    run_case(s, UND_SHORT_SETUP)
    a = s._rectangle_args([nx, ny], "XY", [0.02, 0.03], None, None, [0, 0.01, 20], 0, True)
    o = s._opts("", 112188979912321.0, None, None, 0.01, 24, 0, 0, 0, "mixed")
    n, got = nx * ny, []
    pts, nrm = np.empty(3 * n), np.empty(3 * n)
    assert lib().osc_surface_rectangle(*a, dptr(pts), dptr(nrm), None) == 0
    for rect in (True, False):
        out, lv = torch.full((n,), -1.0, dtype=torch.float64), torch.full((n,), -1, dtype=torch.int32)
        if locked:
            out, lv = out.pin_memory(), lv.pin_memory()
        out, lv, nnc = out.numpy(), lv.numpy(), ctypes.c_longlong()
        tail = (ctypes.byref(o),) + ((None, None) if rect else ()) + (dptr(out), i32ptr(lv), ctypes.byref(nnc))
        if rect:
            s._ctx.call("osc_power_density_rectangle", *a, 0, *tail)
        else:
            s._ctx.call("osc_power_density", dptr(pts), dptr(nrm), n, 0, *tail)
        got.append((out, lv))
    assert got[0][0].min() > 0 and np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


def _stl_both(path, calls):
    out = []
    for o in (sr(gpu=1), OracleSR()):
        run_case(o, UND_SHORT_SETUP)
        o.add_stl(path, translation=[0, 0, 20])
        res = o.calculate_power_density_stl([0, 0, 0], **calls)
        out.append(np.array([r[1] for r in res]))
    return out


# Facets between the trajectory and a plate: few, over one staged tile, and more than a CTA keeps after its cull;
# coplanar, grazing and edge-on ones among them.  Shadowing is the oracle's sample by sample (a lost or an extra
# sample changes a facet by >= 1e-3), the terms are within 1e-12.
@pytest.mark.parametrize("shields, spread, level, seed", [(0, 0.0, 10, 1), (20, 0.006, 11, 2), (90, 0.0003, 9, 3),
                                                           (1100, 0.0002, 4, 4), (12, 0.004, 14, 5)])
def test_stl_shadowing_matches_oracle(tmp_path, shields, spread, level, seed):
    from cases import _grid_plate, _write_stl
    rng = np.random.default_rng(seed)
    tris = _grid_plate(3, 3, -0.012, 0.012, -0.012, 0.012, (0.0, 0.0, 1.0))
    for k in range(shields):
        c = np.array([*rng.normal(0, spread + 1e-4, 2), rng.uniform(-18, -2)])
        depth = [0.0, 0.0, 1.0, 300.0][k % 4]
        p = [tuple(c + rng.normal(0, 0.0015, 3) * np.array([1, 1, depth])) for _ in range(3)]
        tris.append(((0.0, 0.0, -1.0), *p))
    path = str(tmp_path / "mesh.stl")
    _write_stl(path, tris)
    got, want = _stl_both(path, dict(max_level=level))
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


# Device trajectories: one or two ideal undulators in registers, other fields through the general evaluation, one to
# several trajectories a warp.  Every path rounds alike: a job's trajectory does not depend on its company, and an
# undulator given as two halves of its amplitude in one job (registers) or with an idle grid beside them (general
# evaluation) moves the particle the same way.
@pytest.mark.parametrize("npoints", [7, 8, 33, 1000])
def test_device_trajectory_paths_agree_bit_for_bit(npoints):
    from oscars_b200.batch import BatchRunner, Job, grid, undulator
    a = undulator([0, 0.5, 0], [0, 0, 0.05], 5, phase=-0.7, taper=0.01)
    b = undulator([0.25, 0, 0.01], [0, 0, 0.04], 6)
    idle = grid(np.zeros((8, 3)), [2, 2, 2], [5, 5, 5], [1, 1, 1])

    def job(*fields):
        return Job(fields=list(fields), energy_GeV=3.0, ctstartstop=(-4e-4 * npoints, 5e-4 * npoints), npoints=npoints,
                   obs=[[0, 0, 20]], energies_eV=[400.0])
    r = BatchRunner(gpu=0)
    alone = [r.trajectories([job(*f)])[0] for f in ([a], [a, idle], [a, b], [a, b, idle])]
    assert np.array_equal(alone[0], alone[1]) and np.array_equal(alone[2], alone[3])
    many = r.trajectories([job(a), job(a, b), job(a, idle)] * 200)  # 1200 trajectories: three a warp
    for k in range(0, 600, 3):
        assert np.array_equal(many[k], alone[0]) and np.array_equal(many[k + 1], alone[2]) and np.array_equal(many[k + 2], alone[0])


# Batched line tiles (10 energies and more) against the general kernel pinned: same terms, steps and FP32 sums, so the
# same levels and, but for the order of FP64 additions, the same values (1e-10 of the peak, as above).  Tiles that run
# low on active energies hand them on as single entries; jobs below 10 energies sit in the same batch.
@pytest.mark.parametrize("sizes, kw", [([(1, 9), (1, 10), (3, 64), (2, 65)], {}), ([(5, 130), (7, 33), (40, 1), (1, 700)], {}),
                                       ([(4, 40), (1, 12)], dict(max_level=10)), ([(3, 20), (6, 70)], dict(precision=1e-4))])
def test_batch_lines_match_general_kernel(sizes, kw):
    from oscars_b200.batch import BatchRunner, Job, undulator
    jobs = [Job(fields=[undulator([0, 0.5, 0], [0, 0, 0.05], 11, phase=-np.pi / 2)], energy_GeV=3.0, ctstartstop=(-0.5, 0.5),
                npoints=5001, obs=[[1e-4 * k, 5e-5 * k, 20.0 + 0.1 * i] for k in range(m)], energies_eV=np.linspace(300, 1500, n))
            for i, (m, n) in enumerate(sizes)]
    got = []
    for variant in (0, -1):
        r = BatchRunner(gpu=0)
        r.set_variant(variant)
        for _ in range(2):  # the second call replays the captured graph
            f = r.flux(jobs, **kw)
        got.append((f, [x.copy() for x in r.last_levels]))
    for a, b, la, lb in zip(got[0][0], got[1][0], got[0][1], got[1][1]):
        assert np.array_equal(la, lb)
        assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(a))


# The adjoint's forward sums by line tiles against the general kernels pinned (same bounds).
@pytest.mark.parametrize("compute", ["fp64", "mixed"])
@pytest.mark.parametrize("n_obs, n, level", [(1, 10, 9), (3, 65, 10), (5, 33, 7)])
def test_tuning_forward_lines_match_general_kernel(compute, n_obs, n, level):
    from oscars_b200.tuning import TuningProblem
    out = []
    for variant in (0, -1):
        p = TuningProblem(bfield=[0, 0.5, 0], period=[0, 0, 0.05], nperiods=11, obs=[[1e-4 * k, 0, 20.0] for k in range(n_obs)],
                          energies_eV=np.linspace(400, 500, n), level=level, ctstartstop=(-0.5, 0.5), npoints=5001, compute=compute)
        p.sr._ctx.call("osc_set_variant", 2 if compute == "mixed" else 0, variant)
        out.append(p.flux(1 + 0.01 * np.cos(np.arange(22))))
    assert np.max(np.abs(out[0] - out[1])) <= (1e-10 if compute == "mixed" else 1e-12) * np.max(np.abs(out[0]))


# The adjoint's samples take an observer's energies together: observers that change inside, at and across a staged
# chunk (64 or 128 entries).  The gradient is linear in the entries, so it is the sum of the single observers'
# gradients: FP64 to the roundings of 2^10 samples' sums (1e-11), mixed to its FP32 sums over other chunks (1e-5).
@pytest.mark.parametrize("compute, tol", [("fp64", 1e-11), ("mixed", 1e-5)])
@pytest.mark.parametrize("n_obs, n", [(2, 1), (3, 65), (5, 64), (2, 130)])
def test_gradient_is_the_sum_over_observers(compute, tol, n_obs, n):
    from oscars_b200.tuning import TuningProblem
    obs = [[3e-4 * k, 1e-4, 20.0] for k in range(n_obs)]
    s, weight = 1 + 0.01 * np.cos(np.arange(22)), np.cos(np.arange(n_obs * n)).reshape(n_obs, n) + 1.5

    def gradient(o, w):
        p = TuningProblem(bfield=[0, 0.5, 0], period=[0, 0, 0.05], nperiods=11, obs=o, energies_eV=np.linspace(400, 500, n),
                          level=9, ctstartstop=(-0.5, 0.5), npoints=5001, compute=compute)
        return p.vjp(s, w)[1]
    whole = gradient(obs, weight)
    parts = sum(gradient([obs[k]], weight[k:k + 1]) for k in range(n_obs))
    assert np.max(np.abs(whole - parts)) <= tol * np.max(np.abs(whole))


# A beam's trajectories come from host threads that share half trajectories and kept buffers: one particle, more
# particles than slots, and the buffers again at other lengths, against one request per particle of the same
# draw (weights and sums round to 1e-15 a particle).
@pytest.mark.parametrize("method", ["RK4", "RKAS"])
def test_beam_is_the_mean_of_its_particles(method):
    kw = dict(energy_eV=E1_U, npoints=[3, 2], width=[0.004, 0.006], translation=[0, 0, 20], max_level=7, return_numpy=True)
    o = sr(gpu=1)
    o.add_bfield_undulator(bfield=[0, 0.5, 0], period=[0, 0, 0.05], nperiods=5)
    o.set_particle_beam(type="electron", energy_GeV=3, x0=[0, 0, 0], d0=[0, 0, 1], current=0.5, sigma_energy_GeV=0.003,
                        beta=[1.5, 0.8], alpha=[0, 0], emittance=[0.9e-9, 8e-12])
    o.set_ctstartstop(-0.4, 0.4)
    o.set_trajectory_calculation(method, **({} if method == "RK4" else {"precision": 1e-7}))
    for n, points in ((1, 801), (44, 1201), (3, 401)):
        o.set_npoints_trajectory(points)
        o.set_seed(7)
        whole = o.calculate_flux_rectangle(nparticles=n, **kw)[1]
        o.set_seed(7)
        mean = 0
        for _ in range(n):
            o.set_new_particle()
            mean = mean + o.calculate_flux_rectangle(**kw)[1] / n
        # (an RKAS trajectory holds its start time twice: its spline and results are NaN, on both sides)
        assert np.isnan(mean).all() == (method == "RKAS")
        np.testing.assert_allclose(whole, mean, rtol=0, atol=1e-13 * np.max(np.abs(np.nan_to_num(mean))))


# Jobs of uneven trajectory length go in groups, sorted by it, whose waves overlap the longer integrations: against
# each job alone (levels equal; the spans of its sums round in FP64 only).
def test_batch_groups_match_single_jobs():
    from oscars_b200.batch import BatchRunner, Job, undulator
    def job(points, side, n, ct):
        xs = np.linspace(-0.002, 0.002, side)
        return Job(fields=[undulator([0, 0.6, 0], [0, 0, 0.04], 8)], energy_GeV=3, ctstartstop=(-ct, ct), npoints=points,
                   obs=[[x, y, 20.0] for x in xs for y in xs], energies_eV=np.linspace(300, 900, n), current=0.5)
    jobs = [job(9001, 40, 340, 0.5), job(12001, 3, 20, 0.6), job(3001, 41, 330, 0.4), job(10001, 2, 5, 0.5)]
    kw = dict(compute="mixed", max_level=11)
    r = BatchRunner(gpu=0)
    for _ in range(2):  # the second call replays the captured graph
        whole = r.flux(jobs, **kw)
        levels = [x.copy() for x in r.last_levels]
        for k, j in enumerate(jobs):
            one = BatchRunner(gpu=0)
            alone = one.flux([j], **kw)[0]
            assert np.array_equal(levels[k], one.last_levels[0])
            assert np.max(np.abs(whole[k] - alone)) <= 1e-12 * np.max(np.abs(alone))


# The trajectory adjoint's segments of 64 steps, full and ragged, few and many, with other fields beside the tuned one
# (their gradient enters the steps, not the factors), against central differences of the host's trajectory
# (h = 1e-6: roundings 1e-16 / h of the knots and h^2: 1e-5 of the gradient).
@pytest.mark.parametrize("npoints", [66, 129, 640, 1411])
def test_trajectory_gradient_at_segment_edges(npoints):
    from oscars_b200.tuning import TuningProblem
    p = TuningProblem(bfield=[0, 0.5, 0], period=[0, 0, 0.05], nperiods=3, obs=[[0, 0, 20.0]], energies_eV=[400.0], level=4,
                      ctstartstop=(-0.15, 0.11), npoints=npoints)
    p.sr.add_bfield_epu(bfieldA=[0, 0.2, 0], bfieldB=[0.1, 0, 0], period=[0, 0.002, 0.06], nperiods=3, phase=0.4, taper=0.1,
                        frequency=3e8, time_offset=1e-10)
    p.sr.set_npoints_trajectory(npoints)

    def knots(s):
        p.set_scale(s)
        p.sr.calculate_trajectory()
        return p.sr.trajectory_array()[1:]
    s0 = 1 + 0.02 * np.cos(np.arange(6))
    weight = np.random.default_rng(3).standard_normal((9, npoints)) * np.array([1] * 3 + [1e-3] * 3 + [1e-6] * 3)[:, None]
    g = p.trajectory_vjp(s0, weight[:, :knots(s0).shape[1]])
    fd = []
    for e in 1e-6 * np.eye(6):
        k1, k0 = knots(s0 + e), knots(s0 - e)
        fd.append(np.sum(weight[:, :k1.shape[1]] * (k1 - k0)) / 2e-6)
    assert np.linalg.norm(g - np.array(fd)) <= 1e-5 * np.linalg.norm(fd)


# Mixed spectra whose phase steps reach pi at the coarse levels (harmonics up to the 25th at level 9 and 10): the steps
# bounded per quarter chunk settle the stop rule as the general kernel's single ones do, so the levels are the same ones.
@pytest.mark.parametrize("low, high, n", [(400, 12000, 130), (6000, 12000, 33), (200, 300, 64)])
def test_mixed_spectrum_steps_settle_the_same_levels(low, high, n):
    out = []
    for variant in (0, -1):
        s = sr(gpu=1)
        s._ctx.call("osc_set_variant", 2, variant)
        run_case(s, UND_SHORT_SETUP)
        e, f = s.calculate_spectrum(obs=[0.002, 0.001, 20], energy_range_eV=[low, high], npoints=n, compute="mixed",
                                    return_numpy=True)
        out.append((f, s.last_levels.copy()))
    assert np.array_equal(out[0][1], out[1][1])
    assert np.max(np.abs(out[0][0] - out[1][0])) <= 1e-10 * np.max(np.abs(out[0][0]))


# The block-parallel splines against the serial sweeps at the edges of their chunks (56 points and more, 512 threads): a
# chunk's entering value keeps less than 2^-56 of any start, and a difference of an ulp in a factor or a right side moves
# its neighbours by less than twice that: a few 1e-16 of the largest second derivative, 1e-14.
@pytest.mark.parametrize("npoints", [5, 57, 58, 59, 60, 114, 115, 28674, 28675, 60001])
def test_block_parallel_splines_match_serial_sweeps(npoints):
    from oscars_b200.batch import BatchRunner, Job, undulator
    job = Job(fields=[undulator([0.1, 0.5, 0], [0, 0, 0.05], 12, phase=-0.7)], energy_GeV=3.0, ctstartstop=(-4e-4 * npoints, 5e-4 * npoints),
              npoints=npoints, obs=[[0, 0, 20]], energies_eV=[400.0])
    got = []
    for kernel in (1, 2):
        r = BatchRunner(gpu=0)
        r.ctx.call("osc_set_batch_spline_kernel", kernel)
        got.append(r.trajectories([job])[0])
    assert np.array_equal(got[0][:10], got[1][:10])
    scale = np.max(np.abs(got[0][10:]), axis=1, keepdims=True)
    assert np.all(np.abs(got[0][10:] - got[1][10:]) <= 1e-14 * scale)
