"""The host runtime's random numbers are those of the Python definition, for every seed and index."""
import numpy as np
import pytest

from blackwellllm_b200.sampling.params import SamplingParams, row_draws, uniform, uniform_many


@pytest.mark.parametrize("seeds,indices", [([], []), ([0], [0]), ([-1, 1 << 63, (1 << 70) + 5, 2 ** 32], [1, 2 ** 32 + 7, 2 ** 64 + 3, 0])])
def test_uniform_many(seeds, indices):
    got = uniform_many(seeds, indices)
    assert got.dtype == np.float32 and got.tolist() == [uniform(s, i) for s, i in zip(seeds, indices)]


@pytest.mark.parametrize("seeds,indices", [([5, 5, 5], [0]), ([5], [0, 1]), ([], [0])])
def test_uniform_many_refuses_unequal_lengths(seeds, indices):
    with pytest.raises(ValueError):
        uniform_many(seeds, indices)


def test_uniform_many_takes_whole_numbers_only():
    assert uniform_many(np.array([7, -1]), np.array([3, 4])).tolist() == [uniform(7, 3), uniform(-1, 4)]
    for bad in (1.5, None, "1"):
        with pytest.raises(TypeError):
            uniform_many([bad], [0])


def test_rows_draw_from_their_own_streams():
    greedy, warm = SamplingParams(temperature=0.0), SamplingParams(temperature=0.6)
    # a greedy row's seed and index are not looked at, and rows beyond the last are nobody's
    got = row_draws([greedy, warm, greedy, warm], [None, 5, "x", 6, 7], [None, 2, None, 9, 1])
    assert got.dtype == np.float32 and got.tolist() == [0.0, uniform(5, 2), 0.0, uniform(6, 9)]
    assert row_draws([warm, greedy], [5], [2]).tolist() == [uniform(5, 2), 0.0]
    for seeds, indices in (([5], [0, 1, 2]), ([5, 6, 7], [0])):      # one seed is not every row's
        with pytest.raises(IndexError):
            row_draws([warm] * 3, seeds, indices)
    with pytest.raises(TypeError):
        row_draws([warm], [None], [0])
