"""FP64 products on Brick8 matrices of more slices than one wave holds with two slots in flight
(8 per SM), which take one slot at a time: on both sides of that line on 148 SMs (37,888 nodes),
the last slice and block ragged.  Bound as in test_spmv_split_gpu."""
import pytest

from test_spmv_split_gpu import test_spmv_split as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(36, 31, 31), (36, 31, 32), (40, 33, 29)])
def test_one_slot_in_flight(cells):
    check("brick8", cells, "f64")
