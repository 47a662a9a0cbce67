"""Gaussian sketches whose last variate falls around the end of a batch of generator words."""
import numpy as np
import pytest

from oracle.rng import gaussian_matrix

pytestmark = pytest.mark.gpu


# a batch of 681 attempts yields about 1070 variates (681 * pi / 4 * 2)
@pytest.mark.parametrize("seed", [1, 77, 4000000000])
@pytest.mark.parametrize("n", [2, 681, 1361, 1363, 2140, 6421])
def test_sketch_lengths(lib, n, seed):
    got, ref = lib.gaussian_sketch(n, 1, seed), gaussian_matrix(n, 1, seed)
    # the device log may round differently in the last place
    assert np.max(np.abs(got - ref) / np.maximum(np.abs(ref), 1e-300)) < 4 * np.finfo(float).eps


def test_every_length_near_a_batch(lib):
    ref = gaussian_matrix(1200, 1, 9)
    for n in range(1030, 1110):
        got = lib.gaussian_sketch(n, 1, 9)
        assert np.max(np.abs(got - ref[:n]) / np.maximum(np.abs(ref[:n]), 1e-300)) < 4 * np.finfo(float).eps
