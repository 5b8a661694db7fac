"""FP64 H*x on sectors with identity blocks and ragged tiles: patch sizes at
the edges of the 8-wide MMA blocks and of the 32- and 64-wide tiles, left and
right sizes unlike, in every tile configuration and the default one, against
the oracle; and the device Lanczos on sectors around its chunk lengths."""
import numpy as np
import pytest

from dmrgpp_b200 import superblock as sb

pytestmark = pytest.mark.gpu

SIZES = [([1], [1]), ([7, 8, 9], [1, 16, 5]), ([31, 32, 33], [33, 31, 32]), ([63, 64, 65], [8, 65, 63]),
         ([130, 3, 64], [70, 129, 1])]


@pytest.mark.parametrize("left,right", SIZES)
def test_identity_terms_and_ragged_tiles(cuda_lib, cuda_device, oracle_built, left, right):
    from dmrgpp_b200 import plugin
    prob = sb.spin_chain_like(left, right, seed=5 + len(left) + left[0])
    x = np.random.default_rng(3).standard_normal(prob.dim)
    ref = oracle_built.kron_apply(prob, x)
    bg = plugin.BatchedGemm.from_problem(prob)
    assert bg.f_alg == prob.flops()          # identity blocks still counted dense
    scale = np.abs(ref).max()
    assert np.abs(bg(x) - ref).max() < 1e-12 * scale
    for cfg in range(8):
        for ipc in (1, 4):
            bg.set_config(cfg, ipc)
            assert np.abs(bg(x) - ref).max() < 1e-12 * scale, (cfg, ipc)
    bg.close()


# rows around one chunk of the projections (512), odd and even; six blocks of
# one chunk (several chunks a block: test_lanczos_chunks_gpu.py)
@pytest.mark.parametrize("left,right", [([511], [1]), ([512], [1]), ([513], [1]), ([32, 33], [32, 31]), ([60], [51])])
def test_lanczos_chunk_edges(cuda_lib, cuda_device, left, right):
    from dmrgpp_b200 import plugin
    prob = sb.spin_chain_like(left, right, seed=11)
    bg = plugin.BatchedGemm.from_problem(prob)
    init = np.random.default_rng(2).standard_normal(prob.dim)
    H = prob.dense() if prob.dim <= 2100 else None
    e, z, _ = bg.lanczos_lowest(init, steps=200, tolerance=1e-13)
    assert abs(np.linalg.norm(z) - 1.0) < 1e-12
    hz = bg(z)
    assert abs(z @ hz - e) < 1e-11 * abs(e)
    if H is not None:
        w = np.linalg.eigvalsh(H)
        assert abs(e - w[0]) < 1e-11 * abs(w[0])
    bg.close()
