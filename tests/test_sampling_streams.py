"""The host runtime's random numbers are those of the Python definition, for every seed and index."""
import numpy as np
import pytest

from blackwellllm_b200.sampling.params import uniform, uniform_many


@pytest.mark.parametrize("seeds,indices", [([], []), ([0], [0]), ([-1, 1 << 63, (1 << 70) + 5, 2 ** 32], [1, 2 ** 32 + 7, 2 ** 64 + 3, 0])])
def test_uniform_many(seeds, indices):
    got = uniform_many(seeds, indices)
    assert got.dtype == np.float32 and got.tolist() == [uniform(s, i) for s, i in zip(seeds, indices)]
