"""y = H x with y over x (the same buffer, or shifted by some elements): what
separate buffers give.  The sectors hold terms with an identity factor, whose
one product reads X in the launch that writes Y, so an apply that does not
look for the overlap races."""
import ctypes

import numpy as np
import pytest

from dmrgpp_b200 import superblock as sb

pytestmark = pytest.mark.gpu


def _far(n=800, l=16, r=33):
    """One term with an identity factor that couples patches n / 2 apart: more
    output tiles than run at once, the later of which read what the earlier
    ones have written over."""
    rng = np.random.default_rng(6)
    eye = np.asfortranarray(np.eye(l))
    A = {(i, (i + n // 2) % n, 0): eye for i in range(n)}
    B = {k: np.asfortranarray(rng.standard_normal((r, r))) for k in A}
    return sb.KronProblem(np.full(n, l), np.full(n, r), 1, A, B)


SECTORS = {"small": lambda: sb.spin_chain_like([9, 33, 17], [12, 40, 7], seed=4),
           "microbench": lambda: sb.c2_problem(seed=3),
           "wide": lambda: sb.spin_chain_like([200, 420, 200], [180, 400, 210], seed=5),
           "far": _far}
SHIFTS = [0, 1, 64, -3]


def _buffers(x, shift):
    """One buffer that holds x, and y's view of it `shift` elements on."""
    import torch
    n, at = x.size, max(0, -shift)
    buf = torch.zeros(n + abs(shift), dtype=torch.from_numpy(x).dtype, device="cuda")
    xv, yv = buf[at:at + n], buf[at + shift:at + shift + n]
    xv.copy_(torch.from_numpy(x))
    return xv, yv


def _check(apply, x, ref, tol):
    import torch
    for shift in SHIFTS:
        for _ in range(3):
            xv, yv = _buffers(x, shift)
            apply(xv, yv)
            torch.cuda.synchronize()
            y = yv.cpu().numpy()
            assert np.abs(y - ref).max() <= tol * np.abs(ref).max(), shift


@pytest.mark.parametrize("name", sorted(SECTORS))
def test_apply_over_its_input(cuda_lib, cuda_device, name):
    """Default configuration, every other one, and the tensor-core form; equal
    to the same form on separate buffers up to the order of its sums."""
    from dmrgpp_b200 import plugin
    prob = SECTORS[name]()
    x = np.random.default_rng(1).standard_normal(prob.dim)
    bg = plugin.BatchedGemm.from_problem(prob, precision=plugin.TF32X3)
    y3 = bg(x)
    _check(bg.apply_Htarget, x, y3, 0.0)
    bg.set_precision(plugin.FP64)
    ref = bg(x)
    _check(bg.apply_Htarget, x, ref, 1e-13)
    for cfg in range(8):
        bg.set_config(cfg, 2)
        _check(bg.apply_Htarget, x, ref, 1e-13)
    bg.close()


def test_complex_apply_over_its_input(cuda_lib, cuda_device):
    from dmrgpp_b200 import plugin
    prob = SECTORS["small"]()
    rng = np.random.default_rng(2)
    A = {k: np.asfortranarray(m + 1j * rng.standard_normal(m.shape)) for k, m in prob.A.items()}
    B = {k: np.asfortranarray(m.astype(np.complex128)) for k, m in prob.B.items()}
    bg = plugin.BatchedGemm.from_problem(sb.KronProblem(prob.lsz, prob.rsz, prob.noperator, A, B))
    x = rng.standard_normal(prob.dim) + 1j * rng.standard_normal(prob.dim)
    _check(bg.apply_Htarget, x, bg(x), 1e-13)
    bg.close()


@pytest.mark.parametrize("name", ["small", "microbench", "far"])
def test_noalloc_over_its_input(cuda_lib, cuda_device, name):
    import torch
    from dmrgpp_b200 import _capi, plugin
    prob = SECTORS[name]()
    x = np.random.default_rng(3).standard_normal(prob.dim)
    bg = plugin.BatchedGemm.from_problem(prob)
    ref = bg(x)
    bg.close()
    A, ldA, B, ldB = prob.tables()
    t = plugin._DescTables(prob.noperator, prob.npatches, prob.lsz, prob.rsz, A, ldA, B, ldB, 0,
                           torch.cuda.current_stream().cuda_stream, -1)

    def apply(xv, yv):
        rc = cuda_lib.dmrgpp_kron_apply_noalloc(ctypes.byref(t.desc), ctypes.c_void_p(xv.data_ptr()),
                                                ctypes.c_void_p(yv.data_ptr()))
        assert rc == _capi.OK, cuda_lib.dmrgpp_kron_noalloc_last_error()

    _check(apply, x, ref, 1e-13)
