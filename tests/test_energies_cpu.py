"""Photon energies given point by point: what float() makes of each, whatever holds them."""
import array
import decimal
import fractions

import numpy as np
import pytest
import torch

from oscars_b200.sr import sr

CASES = [
    [1.0, 2.5], (1, 2, True), [2 ** 70, 1], ["1", " 2e3 "], "123", b"12", range(4), {3.0: 1}, array.array("f", [1.5, 2.5]),
    [fractions.Fraction(1, 3), decimal.Decimal("0.1")], [np.float32(0.1), 0.1], [None, 1.0], [1 + 0j], [10 ** 400], [[1.0], [2.0]],
    np.linspace(1, 2, 7)[::3], np.arange(4.0)[::-1], np.arange(4, dtype=">i4"), np.arange(3, dtype=np.float16), np.arange(3, dtype=np.longdouble) / 3,
    np.array(["1", "2"]), np.array([1, "2"], dtype=object), np.array([1 + 0j]), np.array([[1.0], [2.0]]), np.matrix([1.0, 2.0]),
    np.array([(1.0,)], dtype=[("a", "f8")]), np.array(["2020-01-01"], dtype="M8[D]"), np.array([5], dtype="m8[s]"),
    [np.datetime64("2020-01-01")], np.ma.array([1.0, 2.0], mask=[0, 1]), [1.0, np.ma.masked], [float("nan"), 1.0],
    torch.tensor([1.0, 2.0]), torch.tensor([1.0, 2.0], requires_grad=True), torch.tensor([1.0], dtype=torch.bfloat16),
    [torch.tensor(1.0, requires_grad=True), 2.0],
]


@pytest.mark.parametrize("points", CASES, ids=lambda v: type(v).__name__)
@pytest.mark.filterwarnings("ignore")
def test_energy_points_are_floats_of_the_elements(points):
    def outcome(f):
        try:
            return f()
        except Exception as e:
            return type(e)
    want = outcome(lambda: np.array([float(e) for e in points]))
    got = outcome(lambda: sr._energies(0, None, points))
    if isinstance(want, type):
        assert got is want
        return
    assert got.dtype == np.float64 and got.flags.c_contiguous and np.array_equal(got, want, equal_nan=True)
    assert not np.shares_memory(got, points) if isinstance(points, np.ndarray) else True
