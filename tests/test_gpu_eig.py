"""Device Davidson eigensolver (lobpcg_serial.solve) against the golden KATs and the oracle.

Eigenvalue tolerance 1e-7 Ry (the plain-FP64 parity bar), with the solver run at tol 1e-9."""
import json
import os

import numpy as np
import pytest

from oracle import lobpcg
from tests.helpers import kproblem, make_context

pytestmark = pytest.mark.gpu


def _diag_context(dz, diag):
    """A context whose H is diag(values): kinetic = diag, V(r) = 0, no projectors."""
    n = len(diag)
    hkl = np.array([[i, 0, 0] for i in range(n)], dtype=np.int32)
    kc = dz.KpointContext(8, 4, 4, 1.0, hkl, np.asarray(diag, float), np.zeros((n, 3)))
    kc.set_vloc(np.zeros(8 * 4 * 4))
    return kc


@pytest.mark.parametrize("case", range(2))
def test_lobpcg_diagonal_kats(dz, case):
    with open(os.path.join(os.path.dirname(__file__), "golden", "lobpcg_diag.json")) as f:
        doc = json.load(f)["cases"][case]
    kc = _diag_context(dz, doc["diag"])
    r = kc.hermitian_eigen_decomp_iterative(np.array(doc["diag"]), doc["nbands"], dz.Options(max_iter=doc["max_iter"], tol=doc["tol"]))
    assert np.abs(r.values - np.array(doc["expected"])).max() < doc["atol"]
    kc.close()


@pytest.mark.parametrize("diag,nbands", [([0.0], 1), ([0.0] * 4, 2), ([0.0, 0.0, 1.0], 3)])
def test_operator_with_zero_levels(dz, diag, nbands):
    """One plane wave at Gamma, and subspaces whose matrix is zero: unit, orthogonal vectors all the same."""
    kc = _diag_context(dz, diag)
    r = kc.hermitian_eigen_decomp_iterative(np.array(diag), nbands, dz.Options(max_iter=20, tol=1e-9))
    assert np.abs(r.values - np.sort(diag)[:nbands]).max() < 1e-12
    assert np.abs(r.vectors.conj() @ r.vectors.T - np.eye(nbands)).max() < 1e-10
    kc.close()


@pytest.mark.parametrize("k", [(0.0, 0.0, 0.0), (0.25, 0.125, 0.0), (0.5, 0.25, 0.75)])
def test_si2_eigenvalues_match_oracle(dz, k):
    kp = kproblem("si2", 20.0, k)
    kc = make_context(dz, kp)
    diag = kp.ctx.basis.kinetic
    opts = dict(max_iter=200, tol=1e-9)
    r = kc.hermitian_eigen_decomp_iterative(diag, 8, dz.Options(**opts))
    ref = lobpcg.solve(lobpcg.Operator(kp.ctx.n, kp.ctx.apply_batch), diag, 8, lobpcg.Options(**opts))
    dense = np.linalg.eigvalsh(kp.ctx.dense_hamiltonian())[:8]
    assert r.converged
    assert np.abs(r.values - ref.values).max() < 1e-7
    assert np.abs(r.values - dense).max() < 1e-7
    # Ritz vectors are eigenvectors: ||H v - lambda v|| small, orthonormal.  The solver may stop
    # through the reference's "no vector could be added" exit (serial.zig:269-283): every new
    # direction r/(diag - lambda) fell under the 1e-8 Gram-Schmidt drop norm, so the residual is
    # bounded by 1e-8 * max|diag - lambda| <= 1e-8 * (ecut + |lambda|), not by tol.
    hv = kp.ctx.apply_batch(r.vectors)
    res = np.linalg.norm(hv - r.values[:, None] * r.vectors, axis=1)
    assert res.max() < 1e-8 * (20.0 + np.abs(r.values).max())
    assert abs(res.max() - r.max_residual) < 1e-9
    assert np.abs(r.vectors.conj() @ r.vectors.T - np.eye(8)).max() < 1e-10
    kc.close()


def test_init_diagonal_and_warm_start(dz):
    kp = kproblem("si2", 20.0, (0.25, 0.25, 0.0))
    kc = make_context(dz, kp)
    diag = kp.ctx.basis.kinetic
    dense = np.linalg.eigvalsh(kp.ctx.dense_hamiltonian())[:8]
    r = kc.hermitian_eigen_decomp_iterative(diag, 8, dz.Options(max_iter=200, tol=1e-9, init_diagonal=True))
    assert np.abs(r.values - dense).max() < 1e-7
    # a warm start from converged vectors (KpointCache) needs a small fraction of a cold start's iterations
    r2 = kc.hermitian_eigen_decomp_iterative(diag, 8, dz.Options(max_iter=200, tol=1e-8, init_vectors=r.vectors))
    assert np.abs(r2.values - dense).max() < 1e-7
    assert r2.iterations * 4 <= r.iterations
    kc.close()


def test_al4_twelve_bands(dz):
    """Al4 (metal, 27^3 odd box), 12 bands, default subspace (max_subspace 56, restarts included)."""
    kp = kproblem("al4", 25.0, (0.125, 0.25, 0.375))
    kc = make_context(dz, kp)
    diag = kp.ctx.basis.kinetic
    r = kc.hermitian_eigen_decomp_iterative(diag, 12, dz.Options(max_iter=300, tol=1e-9))
    dense = np.linalg.eigvalsh(kp.ctx.dense_hamiltonian())[:12]
    assert r.converged
    assert np.abs(r.values - dense).max() < 1e-7
    kc.close()


def test_small_subspace_restarts_match_oracle(dz):
    """max_subspace 24 for 8 bands restarts every few iterations (serial.zig:285-293); both the
    device solver and the oracle converge to the dense eigenvalues."""
    kp = kproblem("si2", 20.0, (0.25, 0.25, 0.0))
    kc = make_context(dz, kp)
    diag = kp.ctx.basis.kinetic
    opts = dict(max_iter=400, tol=1e-9, max_subspace=24)
    r = kc.hermitian_eigen_decomp_iterative(diag, 8, dz.Options(**opts))
    ref = lobpcg.solve(lobpcg.Operator(kp.ctx.n, kp.ctx.apply_batch), diag, 8, lobpcg.Options(**opts))
    dense = np.linalg.eigvalsh(kp.ctx.dense_hamiltonian())[:8]
    assert r.converged and ref.converged
    assert np.abs(r.values - dense).max() < 1e-7
    assert np.abs(r.values - ref.values).max() < 1e-7
    kc.close()


def test_not_converged_returns_best_estimate(dz):
    """serial.zig:298-306: no error when max_iter runs out; the last Ritz values come back."""
    kp = kproblem("si2", 20.0)
    kc = make_context(dz, kp)
    r = kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, 8, dz.Options(max_iter=1, tol=1e-12))
    assert not r.converged and r.iterations == 1
    assert np.all(np.isfinite(r.values))
    kc.close()


def test_batch_matches_independent_solves(dz):
    """dftcuda_eig_solve_batch on k-points with different n_pw (Si8, 751 / 762 / 765 / 740 plane
    waves at 12 Ry) against one dftcuda_eig_solve per k-point: the same iteration counts and
    eigenvalues (the runs share no data; only their order on the GPU differs)."""
    ks = [(0.0, 0.0, 0.0), (0.125, 0.25, 0.0), (0.375, 0.125, 0.25), (0.5, 0.5, 0.25)]
    kps = [kproblem("si8", 12.0, k) for k in ks]
    assert len({kp.ctx.n for kp in kps}) > 1
    opts = dict(max_iter=200, tol=1e-8)
    nb = 16
    single = []
    for kp in kps:
        kc = make_context(dz, kp)
        single.append(kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, nb, dz.Options(**opts)))
        kc.close()
    ctxs = [make_context(dz, kp) for kp in kps]
    batch = dz.hermitian_eigen_decomp_iterative_batch(ctxs, [kp.ctx.basis.kinetic for kp in kps], nb, dz.Options(**opts))
    for kc in ctxs:
        kc.close()
    for a, b, kp in zip(single, batch, kps):
        assert b.converged
        assert a.iterations == b.iterations and a.h_applies == b.h_applies
        assert np.abs(a.values - b.values).max() < 1e-12
        dense = np.linalg.eigvalsh(kp.ctx.dense_hamiltonian())[:nb]
        assert np.abs(b.values - dense).max() < 1e-7


NO_THREADS = """
import ctypes, sys
sys.path.insert(0, {root!r})
import dftzig_loader
from tests.helpers import kproblem, make_context
dz = dftzig_loader.load()
kps = [kproblem("si2", 10.0, (0.1 * i, 0.25, 0.0)) for i in range(4)]
ctxs = [make_context(dz, kp) for kp in kps]
kin = [kp.ctx.basis.kinetic for kp in kps]
first = dz.hermitian_eigen_decomp_iterative_batch(ctxs, kin, 4)
libc = ctypes.CDLL(None)
attr = ctypes.create_string_buffer(256)
libc.pthread_attr_init(attr)
libc.pthread_attr_setstacksize(attr, ctypes.c_size_t(1 << 46))  # more than there is address space for
assert libc.pthread_setattr_default_np(attr) == 0
again = dz.hermitian_eigen_decomp_iterative_batch(ctxs, kin, 4)
assert max(abs(a.values - b.values).max() for a, b in zip(first, again)) < 1e-9
"""


def test_batch_without_threads_to_start():
    """Where the host has no thread to give, the batch is issued with those it has (in a process of its own: the default
    stack size that keeps threads from starting is the process's)."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", NO_THREADS.format(root=root)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_profile_of_a_batch_counts_each_run_alone(dz):
    """A batch's runs are issued by several host threads: each context's profile counts its own launches."""
    kps = [kproblem("si8", 12.0, (0.1 * i, 0.25, 0.0)) for i in range(6)]
    opts = dz.Options(max_iter=5, tol=1e-12)

    def launches(batches):
        ctxs = [make_context(dz, kp) for kp in kps]
        for kc in ctxs:
            kc.set_profiling()
        for at in batches:
            dz.hermitian_eigen_decomp_iterative_batch([ctxs[i] for i in at], [kps[i].ctx.basis.kinetic for i in at], 16, opts)
        got = [kc.profile()["kernel_launches"] for kc in ctxs]
        for kc in ctxs:
            kc.close()
        return got

    assert launches([range(6)]) == launches([[i] for i in range(6)])


def test_large_block_uses_panel_cholesky(dz):
    """100 bands: 104-column Davidson blocks go through the panel Cholesky (GEMM trailing updates);
    eigenvalues against dense diagonalisation."""
    kp = kproblem("si8", 12.0, (0.25, 0.0, 0.0))
    kc = make_context(dz, kp)
    r = kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, 100, dz.Options(max_iter=300, tol=1e-8))
    kc.close()
    dense = np.linalg.eigvalsh(kp.ctx.dense_hamiltonian())[:100]
    assert r.converged
    assert np.abs(r.values - dense).max() < 1e-7
    assert np.abs(r.vectors.conj() @ r.vectors.T - np.eye(100)).max() < 1e-9
