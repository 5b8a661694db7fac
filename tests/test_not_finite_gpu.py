"""The correction solve and the refinements say so when a residual is not a
finite number, and leave the vectors of the last good step."""
import numpy as np
import pytest

from dmrgpp_b200 import superblock as sb

pytestmark = pytest.mark.gpu


def _start(dim, seed):
    import torch
    return torch.from_numpy(np.random.default_rng(seed).standard_normal(dim)).cuda()


def _sector(scale=1.0, seed=6):
    """scale 1e20: finite in FP64, but the product of two blocks and a vector
    is past the largest FP32 number, so the TF32x3 form overflows."""
    prob = sb.spin_chain_dominant(sb.gaussian_sector_sizes(128, 5, 1.0), seed=seed)
    for table in (prob.A, prob.B):
        for k in table:
            table[k] = table[k] * scale
    return prob


@pytest.mark.parametrize("precond", ["none", "jacobi"])
def test_correction_of_not_a_number(cuda_lib, cuda_device, precond):
    import torch
    from dmrgpp_b200 import _capi, plugin
    bg = plugin.BatchedGemm.from_problem(_sector())
    if precond == "jacobi":
        bg.set_correction_preconditioner(_capi.PRECOND_JACOBI)
    u = _start(bg.dim, 1)
    u = u / torch.linalg.vector_norm(u)
    r = _start(bg.dim, 2)
    r = r - torch.dot(u, r) * u
    for value in (float("nan"), float("inf")):
        bad = r.clone()
        bad[bg.dim // 2] = value
        with pytest.raises(_capi.DmrgppError) as ei:
            bg.correction_solve(u, -100.0, bad, max_iterations=20)
        assert ei.value.status == _capi.NOT_CONVERGED
    t, _, res = bg.correction_solve(u, -1e4, r, max_iterations=500, rel_tolerance=1e-8)
    bg.close()
    assert res <= 1e-8 and bool(torch.isfinite(t).all())


@pytest.mark.parametrize("correction", ["none", "jacobi"])
def test_refinement_whose_corrections_overflow(cuda_lib, cuda_device, correction):
    """psi comes back as the refinement found it, normalised."""
    import torch
    from dmrgpp_b200 import _capi, plugin
    bg = plugin.BatchedGemm.from_problem(_sector(1e20), precision=plugin.TF32X3)
    x = _start(bg.dim, 3)
    assert not bool(torch.isfinite(bg(x)).all())
    if correction == "jacobi":
        bg.set_correction_preconditioner(_capi.PRECOND_JACOBI)
    psi = x.clone()
    with pytest.raises(_capi.DmrgppError) as ei:
        bg.refine_lowest(psi, max_outer=12, inner_iterations=40, inner_tolerance=1e-2)
    assert ei.value.status == _capi.NOT_CONVERGED
    want = x / torch.linalg.vector_norm(x)
    assert float(torch.linalg.vector_norm(psi - want)) <= 1e-13
    bg.close()


def test_group_refinement_with_a_sector_of_nan(cuda_lib, cuda_device):
    """That sector is reported as not converged, the other one converges."""
    import torch
    from dmrgpp_b200 import plugin
    probs = [_sector(), _sector(seed=7)]
    bg = plugin.BatchedGemm.from_problems(probs, precision=plugin.TF32X3)
    offs = bg.sector_offsets()
    _, z, _ = bg.lanczos_lowest_group(_start(bg.dim, 4), steps=200, tolerance=1e-5, reortho=False)
    z[offs[0]:offs[1]] = float("nan")
    e, conv, st = bg.refine_lowest_group(z, max_outer=12, tolerance=1e-10, inner_iterations=80,
                                         inner_tolerance=1e-2, raise_on_no_convergence=False)
    bg.close()
    assert conv.tolist() == [False, True]
    assert bool(torch.isfinite(z[offs[1]:]).all())
    one = plugin.BatchedGemm.from_problem(probs[1])
    e1, _, _ = one.lanczos_lowest(_start(one.dim, 5), steps=400, tolerance=1e-12)
    one.close()
    assert abs(e[1] - e1) <= 1e-10 * abs(e1)
