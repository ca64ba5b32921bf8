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
