"""The device's cell order of meshes of up to 4096 cells is sorted in one block (2048 or 4096 entries), of larger
ones in several: the checks of the boundary's orders at the sizes where that changes."""
import pytest

from test_gpu_cell_order import test_arrays_cross_the_boundary_in_the_callers_order as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 2), (23, 89), (32, 64), (3, 683), (63, 65), (64, 64), (17, 241)])
def test_orders_around_one_block(nx, ny):
    check(nx, ny)
