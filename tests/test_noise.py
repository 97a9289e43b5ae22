"""blml_b200.noise draws default_rng(seed).standard_normal's values with any number of threads."""
import numpy as np
import pytest

from blml_b200 import noise


@pytest.mark.parametrize('threads', [2, 3, 8])
@pytest.mark.parametrize('n', [131072, 131073, 500001])
@pytest.mark.parametrize('seed', [0, 1, 12345678901])
def test_pieces_are_the_serial_draws(seed, n, threads):
    parts = noise._pieces(seed, n, threads)
    assert parts is not None
    np.testing.assert_array_equal(np.concatenate(parts), np.random.default_rng(seed).standard_normal(n))


@pytest.mark.parametrize('n', [1, 7, 131071, 131072])
def test_any_length_and_seed(n):
    for seed in (3, np.int64(3), [3, 4]):
        got = np.concatenate(noise.normal_pieces(seed, n, threads=4))
        np.testing.assert_array_equal(got, np.random.default_rng(seed).standard_normal(n))


def test_threads_that_do_not_meet_fall_back(monkeypatch):
    monkeypatch.setattr(noise, '_pieces', lambda *a: None)
    got = np.concatenate(noise.normal_pieces(5, 140000, threads=4))
    np.testing.assert_array_equal(got, np.random.default_rng(5).standard_normal(140000))
