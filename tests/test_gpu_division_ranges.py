"""The quotients that the kernels form without a range test, over the whole range
of operands that the code around them lets through -- no fallback in between:
every bit equals the IEEE division's."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(4))
def test_quotients_without_range_tests(seed):
    from cuda_emd import _native
    assert _native.check_division(5, 100_000_000, seed=seed) == (0, 0, 0)


def test_float_quotients_without_range_tests():
    from cuda_emd import _native
    assert _native.check_division(6, 400_000_000, seed=3) == (0, 0, 0)
