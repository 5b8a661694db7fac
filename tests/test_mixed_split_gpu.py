"""TF32x3 pass-2 tiles cut along K whose last part sums the others, with 1 to
128 rows: the warps share the columns of the rows that exist."""
import numpy as np
import pytest

from dmrgpp_b200 import superblock as sb

pytestmark = pytest.mark.gpu


# rows of the tiles (right group sizes) at the edges of 32 and of a whole tile,
# column counts around chunks of 32, contractions long enough to be cut
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 64, 65, 96, 97, 128, 129])
@pytest.mark.parametrize("cols", [700, 1025])
def test_split_tiles_of_any_height(cuda_lib, cuda_device, oracle_built, rows, cols):
    from dmrgpp_b200 import plugin
    prob = sb.spin_chain_like([cols, 33], [rows, 2], seed=rows)
    x = np.random.default_rng(rows + cols).standard_normal(prob.dim)
    ref = oracle_built.kron_apply(prob, x)
    bg = plugin.BatchedGemm.from_problem(prob, precision=plugin.TF32X3)
    y = bg(x)
    # the bar of the other TF32x3 tests: two 11-bit parts a factor, 32-bit sums
    assert np.abs(y - ref).max() < 2e-5 * np.abs(ref).max()
    for _ in range(3):
        assert np.array_equal(bg(x), y)   # the parts are summed in their order
    bg.close()
