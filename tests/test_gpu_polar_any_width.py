"""The rotation matrix of the optimized product quantizer for widths that are no whole 16 x 16 tiles."""
import pytest

from tests.test_gpu_polar import test_rotation_is_the_polar_factor as _is_the_polar_factor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,m", [(4, 1), (15, 3), (17, 1), (40, 10), (104, 13), (123, 41), (129, 3), (273, 39), (300, 50), (508, 127)])
def test_rotation_is_the_polar_factor_for_any_width(oracle, dim, m):
    _is_the_polar_factor(oracle, dim, m)
