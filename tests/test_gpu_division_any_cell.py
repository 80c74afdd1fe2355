"""The float division by the cell size at cells of every scale, for every
float input: from 2 m on (no power of two) a subnormal quotient can lie on a
rounding boundary, where the product with a rounded reciprocal may fall on
either side; powers of two, the smallest and the largest cells."""
import pytest

from fdtdsarsim_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('cell_size', [2.5, 3.0, 6.1, 47.3, 1.1e3, 1.7e6, 3.3e30, 3.4e38, 0.25, 8.0, 0.1, 1e-10,
                                       2e-38, 1e-42])
def test_float_division_is_exact_for_every_input(cell_size):
    tested, bad = _native.check_cell_division('float32', cell_size)
    assert tested == 2 ** 32
    assert bad == 0
