"""The device Lanczos where a block of its fused update and projections takes
several chunks of rows: above 592 x 512 rows with short chunks, above
592 x 2048 with long ones; even row counts (16-byte loads) and odd ones, last
chunks ragged, steps replayed from a graph and the rest launch by launch."""
import numpy as np
import pytest

from dmrgpp_b200 import superblock as sb

pytestmark = pytest.mark.gpu


def _lanczos(apply, x, steps):
    """The same recurrence from torch operations: beta before the
    reorthogonalisation, one projection on all stored vectors."""
    import torch
    V = [x / torch.linalg.vector_norm(x)]
    alpha, beta = [], []
    for j in range(steps):
        w = apply(V[j])
        alpha.append(float(torch.dot(w, V[j])))
        w = w - alpha[j] * V[j]
        if j:
            w = w - beta[j - 1] * V[j - 1]
        beta.append(float(torch.linalg.vector_norm(w)))
        w = w / beta[j]
        B = torch.stack(V)
        w = w - B.T @ (B @ w)
        V.append(w / torch.linalg.vector_norm(w))
    T = np.diag(alpha) + np.diag(beta[:-1], 1) + np.diag(beta[:-1], -1)
    e, s = np.linalg.eigh(T)
    return e[0], torch.from_numpy(s[:, 0]).cuda() @ torch.stack(V[:steps])


@pytest.mark.parametrize("left,right,patches", [
    (80, 80, 48),       # 307,200 rows: one block in 75 takes a second short chunk
    (79, 77, 51),       # 310,233, odd
    (112, 110, 97),     # 1,195,040: three or four short chunks a block, the last one ragged
    (160, 158, 49),     # 1,238,720: long chunks
    (159, 161, 49),     # 1,254,351: long chunks, odd
])
def test_several_chunks_a_block(cuda_lib, cuda_device, left, right, patches):
    import torch
    from dmrgpp_b200 import plugin
    prob = sb.spin_chain_like([left] * patches, [right] * patches, seed=3)
    assert prob.dim == left * right * patches > 592 * 512
    bg = plugin.BatchedGemm.from_problem(prob)
    x = torch.randn(prob.dim, generator=torch.Generator().manual_seed(5), dtype=torch.float64).cuda()
    # 12 steps: a graph of 8 and three by themselves after the first
    e, z, n = bg.lanczos_lowest(x, steps=12, tolerance=0.0)
    e_ref, z_ref = _lanczos(bg, x, 12)
    bg.close()
    assert n == 11
    # sums of up to 1.3e6 terms in another order: sqrt(n) eps is 2.5e-13; the
    # vector's error is that over the gap to the next Ritz value, which 12 steps
    # on a spectrum without outliers leave at a few hundredths of |H|
    assert abs(e - e_ref) <= 1e-12 * abs(e_ref)
    sign = 1.0 if float(torch.dot(z, z_ref)) > 0 else -1.0
    assert float(torch.linalg.vector_norm(z - sign * z_ref)) <= 1e-11
