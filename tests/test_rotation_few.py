"""The line between the two tilings of the query rotation for few rows (512
dimensions, whole multiples of 16), with the query counts of the tile tests."""
import pytest

import test_rotation_tiles as tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [496, 511, 512, 527])
def test_rotation_at_the_line(dim):
    tiles.test_rotation_tiles(dim)
