"""Failure paths on the GPU, tested without faulting, trapping or hanging the device.

Every device-side wait in the library is bounded.  dftcuda_debug_set_wait_limits makes the subspace
eigensolver's grid barrier wait for an arrival that no block makes, with a short poll budget, so the
wait runs out: the blocks set the error flag and return, the call reports DFTCUDA_ERR_TIMEOUT, and a
normal call afterwards (on the same context) must succeed.  The same for the int8 products' pipeline,
whose second CTA then never reports its copies.  A NaN injected on the host into one
column of psi must come back as a clean status with the NaN confined to that column.
dftcuda_debug_fail_alloc makes one device allocation fail as cudaMalloc does on a full device: the
call reports DFTCUDA_ERR_OUT_OF_MEMORY and the context stays usable.
"""
import numpy as np
import pytest

from tests.helpers import kproblem, make_context, random_block, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture
def limits(dz):
    yield dz.debug_set_wait_limits
    dz.debug_set_wait_limits()  # defaults again, whatever the test did


def _hermitian(n, seed):
    rng = np.random.default_rng(seed)
    a = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    return a + a.conj().T


def test_grid_barrier_timeout_reports_and_recovers(dz, limits):
    a = _hermitian(200, 1)  # 200 >= 96: the tridiagonal solver with its cooperative grid barrier
    limits(4096, True)
    with pytest.raises(dz.Timeout):
        dz.hermitian_eigen_decomp(a, 20)
    limits()
    r = dz.hermitian_eigen_decomp(a, 20)
    ref = np.linalg.eigvalsh(a)[:20]
    assert np.abs(r.values - ref).max() < 1e-10 * np.abs(ref).max()


def test_eigensolver_timeout_leaves_context_usable(dz, limits):
    kp = kproblem("si8", 20.0, (0.25, 0.0, 0.0))
    kc = make_context(dz, kp)
    limits(4096, True)
    with pytest.raises(dz.Timeout):  # 100 bands: the first Rayleigh-Ritz step is 100 x 100
        kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, 100, dz.Options(max_iter=3, tol=1e-6))
    limits()
    r = kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, 100, dz.Options(max_iter=3, tol=1e-6))
    assert np.isfinite(r.values).all()
    x = random_block(kp.ctx.n, 3, 8)
    assert rel_err(kc.apply_hamiltonian_batched(x), kp.ctx.apply_batch(x)) < 1e-11
    kc.close()


def test_nan_in_one_column_is_confined(dz):
    kp = kproblem("si2", 20.0, (0.25, 0.125, 0.0))
    kc = make_context(dz, kp)
    x = random_block(kp.ctx.n, 5, 9)
    bad = x.copy()
    bad[2, 17] = np.nan
    y = kc.apply_hamiltonian_batched(bad)  # a clean status: no exception
    assert not np.isfinite(y[2]).all()
    keep = [0, 1, 3, 4]
    assert rel_err(y[keep], kp.ctx.apply_batch(x[keep])) < 1e-11
    assert rel_err(kc.apply_hamiltonian_batched(x), kp.ctx.apply_batch(x)) < 1e-11  # the context is unharmed
    kc.close()


@pytest.fixture
def fail_alloc(dz):
    yield dz.debug_fail_alloc
    dz.debug_fail_alloc()  # cancel whatever the test planned


@pytest.mark.parametrize("after", [0, 1, 2])
def test_allocation_failure_reports_and_recovers(dz, fail_alloc, after):
    """The after-th device allocation of the first H|psi> call and of the first Davidson solve on a
    fresh context fails: each call raises OutOfMemory, then succeeds on the same context."""
    kp = kproblem("si8", 20.0, (0.25, 0.0, 0.0))
    kc = make_context(dz, kp)
    x = random_block(kp.ctx.n, 6, 4)
    fail_alloc(after)
    with pytest.raises(dz.OutOfMemory):
        kc.apply_hamiltonian_batched(x)
    fail_alloc()
    assert rel_err(kc.apply_hamiltonian_batched(x), kp.ctx.apply_batch(x)) < 1e-11
    opts = dz.Options(max_iter=3, tol=1e-6)
    fail_alloc(after)
    with pytest.raises(dz.OutOfMemory):
        kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, 20, opts)
    fail_alloc()
    r = kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, 20, opts)
    assert np.isfinite(r.values).all()
    x2 = random_block(kp.ctx.n, 3, 5)
    assert rel_err(kc.apply_hamiltonian_batched(x2), kp.ctx.apply_batch(x2)) < 1e-11
    kc.close()


@pytest.mark.parametrize("m", [1, 2, 40, 95, 96, 200, 1300])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_matrix_that_is_not_finite_is_refused(dz, m, value):
    """One bad entry at a size of each reduction: an error instead of eigenpairs, and the next matrix is solved."""
    a = _hermitian(m, 3)
    bad = a.copy()
    bad[m // 3, m - 1 - m // 4] = value
    if m > 1:
        bad[m - 1 - m // 4, m // 3] = value
    with pytest.raises(dz.LapackFailure):
        dz.hermitian_eigen_decomp(bad, min(m, 5))
    assert np.abs(dz.hermitian_eigen_decomp(a, 1).values - np.linalg.eigvalsh(a)[:1]).max() < 1e-11 * max(1.0, np.abs(a).sum(0).max())


@pytest.mark.parametrize("nbands", [20, 100])
def test_solve_with_nan_potential_is_refused(dz, nbands):
    """Subspaces of 24 and of 104 rows: LapackFailure, and the context solves again with the potential set anew."""
    kp = kproblem("si8", 20.0, (0.25, 0.0, 0.0))
    kc = make_context(dz, kp)
    v = kp.ctx.local_r.copy()
    v[5] = np.nan
    kc.set_vloc(v)
    with pytest.raises(dz.LapackFailure):
        kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, nbands, dz.Options(max_iter=3, tol=1e-6))
    kc.set_vloc(kp.ctx.local_r)
    r = kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, nbands, dz.Options(max_iter=3, tol=1e-6))
    assert np.isfinite(r.values).all() and np.isfinite(r.max_residual)
    kc.close()


def test_residue_pipeline_timeout_reports_and_recovers(dz, limits):
    """Every role of the pipeline gives up by itself: one item per pair and several, one CTA pair and all of them."""
    import torch

    gen = torch.Generator().manual_seed(1)
    for M, N, K in ((300, 400, 4000), (700, 500, 9000)):
        a, b = (torch.randn(n, K, dtype=torch.complex128, generator=gen).cuda() for n in (M, N))
        limits(64, True)
        with pytest.raises(dz.Timeout):
            dz.complex_gemm(a, b)
        limits()
        ref = a @ b.T
        assert float((dz.complex_gemm(a, b) - ref).abs().max()) < 1e-13 * float(ref.abs().max()) * K ** 0.5


def test_projector_product_timeout_leaves_context_usable(dz, limits):
    """An H|psi> large enough for the residue form on the projectors."""
    import torch

    kp = kproblem("si8", 25.0, (0.25, 0.0, 0.0))
    kc = make_context(dz, kp)
    n = kp.ctx.n
    pos = np.random.default_rng(2).uniform(0, 10.0, (64, 3))
    phi = np.random.default_rng(3).normal(size=(5, n))
    kc.set_projectors([dz.SpeciesProjectors([0, 0, 1], np.eye(3), phi)], np.zeros(64, dtype=np.int32), pos)
    x = torch.from_numpy(random_block(n, 400, 7)).cuda()
    good = kc.apply_hamiltonian_batched(x, torch.empty_like(x)).clone()
    limits(64, True)
    with pytest.raises(dz.Timeout):
        kc.apply_hamiltonian_batched(x, torch.empty_like(x))
    limits()
    again = kc.apply_hamiltonian_batched(x, torch.empty_like(x))
    assert float((again - good).abs().max()) <= 1e-13 * float(good.abs().max())
    kc.close()
