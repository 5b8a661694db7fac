"""Density-matrix truncation at the edges of its device reduction: group sizes
around the cluster's columns (8), a warp's rows and the bisection's 32
eigenvalues, a group above the shared-memory limit (host reduction), weights
outside the range the reduction works in, low rank and a zero group."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(sizes, rights, psi, keep):
    import torch
    from dmrgpp_b200 import truncation
    return truncation.density_truncate(sizes, rights, np.arange(len(sizes)), sizes, 0,
                                       torch.from_numpy(psi).cuda(), keep)


def _check(sizes, rights, psi, keep):
    t = _run(sizes, rights, psi, keep)
    assert t["kept_total"] == keep and int(np.sum(t["kept"])) == keep
    off = 0
    for g, (n, r) in enumerate(zip(sizes, rights)):
        M = psi[off:off + n * r].reshape(n, r)
        off += n * r
        rho = M @ M.T
        norm = np.abs(rho).sum(axis=1).max()
        w = t["eigenvalues"][g]
        assert np.all(np.diff(w) >= 0)
        # backward error of the reduction and the bisection: a few n eps |rho|
        assert np.abs(w - np.linalg.eigvalsh(rho)).max() <= 1e-14 * max(n, 8) * norm
        k = int(t["kept"][g])
        V = t["vectors"][g]
        assert V.shape == (n, k)
        if k:
            assert np.abs(V.T @ V - np.eye(k)).max() < 1e-12
            assert np.abs(rho @ V - V * w[n - k:]).max() <= 1e-14 * max(n, 8) * norm


@pytest.mark.parametrize("sizes", [[1], [2, 1], [3, 7, 8, 9], [31, 32, 33], [63, 64, 65, 16], [257, 128], [513, 5]])
def test_group_sizes(cuda_lib, cuda_device, sizes):
    rng = np.random.default_rng(len(sizes) + sizes[0])
    rights = [n + 3 for n in sizes]
    psi = np.concatenate([rng.standard_normal(n * r) for n, r in zip(sizes, rights)])
    _check(sizes, rights, psi / np.linalg.norm(psi), max(1, sum(sizes) // 3))


def test_many_small_groups(cuda_lib, cuda_device):
    """More clusters than run at once, most of their CTAs without a column:
    a CTA reaches its first store to the others' shared memory at once."""
    rng = np.random.default_rng(9)
    sizes = [int(n) for n in rng.integers(1, 10, 900)]
    rights = [int(n) for n in rng.integers(1, 12, 900)]
    psi = np.concatenate([rng.standard_normal(n * r) for n, r in zip(sizes, rights)])
    _check(sizes, rights, psi / np.linalg.norm(psi), sum(sizes) // 2)


@pytest.mark.parametrize("weight", [1e-14, 1e-60, 1e60])
def test_weights_outside_the_reductions_range(cuda_lib, cuda_device, weight):
    rng = np.random.default_rng(4)
    sizes, rights = [40, 33], [50, 44]
    psi = np.concatenate([rng.standard_normal(n * r) for n, r in zip(sizes, rights)]) * weight
    _check(sizes, rights, psi, 30)


def test_low_rank_and_zero_groups(cuda_lib, cuda_device):
    rng = np.random.default_rng(5)
    sizes, rights = [50, 20, 34], [6, 20, 40]     # rank 6, zero, full
    parts = [rng.standard_normal(n * r) for n, r in zip(sizes, rights)]
    parts[1][:] = 0.0
    _check(sizes, rights, np.concatenate(parts), 16)


def test_not_a_number_is_refused(cuda_lib, cuda_device):
    from dmrgpp_b200 import _capi
    psi = np.random.default_rng(6).standard_normal(12 * 12)
    psi[17] = np.nan
    with pytest.raises(_capi.DmrgppError) as ei:
        _run([12], [12], psi, 4)
    assert ei.value.status == _capi.NOT_CONVERGED


def test_group_above_the_device_limit(cuda_lib, cuda_device):
    rng = np.random.default_rng(7)
    sizes, rights = [2049, 9], [40, 12]
    psi = np.concatenate([rng.standard_normal(n * r) for n, r in zip(sizes, rights)])
    _check(sizes, rights, psi / np.linalg.norm(psi), 20)


def test_groups_on_both_sides_of_the_device_limit(cuda_lib, cuda_device):
    """The device's largest group beside one for the host, and small ones."""
    rng = np.random.default_rng(8)
    sizes, rights = [300, 2049, 31, 2048, 1], [310, 60, 40, 70, 3]
    psi = np.concatenate([rng.standard_normal(n * r) for n, r in zip(sizes, rights)])
    _check(sizes, rights, psi / np.linalg.norm(psi), 200)


def test_phase_times_belong_to_their_phases(cuda_lib, cuda_device):
    """A density matrix of 16 states from 2^21 columns: its product takes one
    CTA milliseconds, its reduction and eigenvalues a fraction of one."""
    import torch
    from dmrgpp_b200 import truncation
    n, r = 16, 1 << 21
    psi = torch.randn(n * r, dtype=torch.float64, device="cuda")
    psi /= torch.linalg.vector_norm(psi)
    for _ in range(2):
        truncation.density_truncate([n], [r], np.arange(1), [n], 0, psi, 4)
    t = truncation.truncation_profile()
    assert t["rho"] > 2.0 * t["eigenvalues"]
    assert sum(v for k, v in t.items() if k != "total") <= t["total"] * (1 + 1e-9)
