"""Q4_K and Q5_K prompt products whose column tiles are of 64 columns and just beyond, alone and beside whole ones: a short tile takes two mins
accumulators in turn, a wider one the whole of both. (the bound: `gpu_util.check_sums`)"""
import pytest

import arcint_b200 as A
from gpu_util import check_sums as check, normal_data as data

pytestmark = pytest.mark.gpu


# several units a block (row tiles x column tiles > 148), one, three and five super-blocks a unit
@pytest.mark.parametrize("t", [A.Q4_K, A.Q5_K])
@pytest.mark.parametrize("m,k,n", [(128 * 150, 256, 64), (128 * 150, 768, 65), (128 * 100, 768, 128 + 64), (128 * 100, 256, 128 + 65), (128 * 100, 1280, 128 + 9)])
def test_short_and_whole_tiles(t, m, k, n):
    w, x = data(t, m, k, n, 31 + n)
    with A.Context(0) as c:
        c.stats_reset()
        got = c.run_mul_mat(t, w, k, x)
        assert c.stats().get("gemm_tc", 0) == 1
    check(got, t, w, k, x)
