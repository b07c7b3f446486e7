"""tlq_softfp.cuh's square root with its seed moved by 3 ulps: the GPU's
reciprocal square root may be off by 2^-22.9, 2.14 ulps of a value just below
1, which with the rounding of the host's own seed reaches 2.64."""
import numpy as np
import pytest

from tests.test_softfp import operands, soft  # noqa: F401 (a fixture)


@pytest.mark.parametrize("ulp", [-3, 3])
def test_sqrt_with_the_seeds_full_error(soft, ulp):  # noqa: F811
    g = np.random.default_rng(9)
    one = np.float64(1.0).view(np.uint64)
    near = (one + g.integers(0, 1 << 40, 300_000, dtype=np.uint64)).view(np.float64)  # seeds just below 1
    a = np.concatenate([near, 2.0 * near, 4.0 - near, np.abs(operands(300_000, 5, False)), np.abs(operands(300_000, 6, True))])
    got, want = soft(1, ulp, a, np.ones_like(a)), np.sqrt(a)
    np.testing.assert_array_equal(got.view(np.uint64), want.view(np.uint64))
