"""The solvers start from their inputs alone: buffers that an earlier solve left
full of NaN (the same handle's here, or another's, whose memory the pool hands
on) change nothing.  A first direction formed as z + 0 p, with p not written
yet, turned the solution into NaN.  The energies are compared at the solve's
own tolerance, everything else bit for bit."""
import numpy as np
import pytest

from dmrgpp_b200 import superblock as sb

pytestmark = pytest.mark.gpu


def _sector():
    return sb.spin_chain_dominant(sb.gaussian_sector_sizes(256, 7, 1.4), seed=6)


def _start(dim, seed):
    import torch
    return torch.from_numpy(np.random.default_rng(seed).standard_normal(dim)).cuda()


def _ignoring_the_status(call):
    from dmrgpp_b200 import _capi
    try:
        call()
    except _capi.DmrgppError:
        pass


def _equation(bg, prob):
    """u near the lowest state, its Rayleigh quotient and residual."""
    import torch
    _, z, _ = bg.lanczos_lowest(_start(prob.dim, 3), steps=300, tolerance=1e-12)
    g = _start(prob.dim, 4)
    u = z + 0.05 * g / torch.linalg.vector_norm(g)
    u = u / torch.linalg.vector_norm(u)
    hu = torch.empty_like(u)
    bg.apply_Htarget(u, hu)
    theta = float(torch.dot(u, hu))
    return u, theta, hu - theta * u


@pytest.mark.parametrize("precond", ["none", "jacobi"])
def test_correction_after_not_a_number(cuda_lib, cuda_device, precond):
    """The same handle solves with a residual of NaN, which fills its buffers,
    and then the real equation: bit for bit what a fresh handle returns."""
    import torch
    from dmrgpp_b200 import _capi, plugin
    prob = _sector()
    got = []
    for poison in (False, True):
        bg = plugin.BatchedGemm.from_problem(prob)
        if precond == "jacobi":
            bg.set_correction_preconditioner(_capi.PRECOND_JACOBI)
        u, theta, r = _equation(bg, prob)
        if poison:
            bad = torch.full_like(r, float("nan"))
            _ignoring_the_status(lambda: bg.correction_solve(u, theta, bad, max_iterations=8))
        t, _, res = bg.correction_solve(u, theta, r, max_iterations=3000, rel_tolerance=1e-10)
        bg.close()
        assert res <= 1e-10
        got.append(t)
    assert bool(torch.isfinite(got[1]).all())
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("correction", ["none", "jacobi"])
def test_solve_after_not_a_number(cuda_lib, cuda_device, correction):
    """A whole mixed solve on a handle whose buffers hold NaN."""
    import torch
    from dmrgpp_b200 import _capi, plugin
    prob = _sector()
    x = _start(prob.dim, 9)
    bg = plugin.BatchedGemm.from_problem(prob, precision=plugin.TF32X3)
    bg.set_precision(plugin.FP64)
    e_ref, z, _ = bg.lanczos_lowest(x, steps=400, tolerance=1e-12)
    bg.set_precision(plugin.TF32X3)
    bg.set_correction_preconditioner(_capi.PRECOND_JACOBI)
    bad = torch.full_like(x, float("nan"))
    _ignoring_the_status(lambda: bg.lanczos_lowest(bad, steps=40, reortho=False))
    _ignoring_the_status(lambda: bg.refine_lowest(bad.clone()))
    _ignoring_the_status(lambda: bg.correction_solve(z, e_ref, bad, max_iterations=8))
    bg.set_correction_preconditioner(_capi.PRECOND_NONE)
    e, z, st = bg.solve_lowest(x, tolerance=1e-10, method="mixed", correction=correction)
    bg.close()
    assert st["converged"] and st["fallback"] == 0
    assert bool(torch.isfinite(z).all())
    assert abs(e - e_ref) <= 1e-10 * abs(e_ref)


@pytest.mark.parametrize("correction", ["none", "jacobi"])
def test_group_solve_after_not_a_number(cuda_lib, cuda_device, correction):
    """The group solver's buffers likewise, on one handle."""
    import torch
    from dmrgpp_b200 import _capi, plugin
    probs = [_sector(), sb.spin_chain_dominant(sb.gaussian_sector_sizes(128, 5, 1.0), seed=7)]
    bg = plugin.BatchedGemm.from_problems(probs, precision=plugin.TF32X3)
    x = _start(bg.dim, 9)
    e_ref, z_ref, _ = bg.solve_lowest_group(x, correction=correction)
    bg.set_correction_preconditioner(_capi.PRECOND_JACOBI)
    bad = torch.full_like(x, float("nan"))
    _ignoring_the_status(lambda: bg.refine_lowest_group(bad))
    bg.set_correction_preconditioner(_capi.PRECOND_NONE)
    e, z, st = bg.solve_lowest_group(x, correction=correction)
    bg.close()
    assert np.array_equal(e, e_ref) and torch.equal(z, z_ref)
