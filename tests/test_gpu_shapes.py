"""The edges of the size rules: every four-step box length in both layouts, the packing of the density's
bands, the FFT's axis lengths, and the subspace and Gram matrix sizes at which the eigensolver's kernels
change."""
import numpy as np
import pytest

from oracle import density as odens
from oracle import fft as offt
from oracle.apply import ApplyContext
from oracle.pw import Basis, Grid
from tests.helpers import kproblem, make_context, random_block, rel_err

pytestmark = pytest.mark.gpu

LENGTHS = [20, 24, 27, 30, 32, 36, 40, 45, 48, 60, 64, 72, 75, 80, 90, 96, 100, 108, 120, 128]


def _sphere(n, r):
    h = np.arange(-r, r + 1)
    hkl = np.stack(np.meshgrid(h, h, h, indexing="ij"), -1).reshape(-1, 3).astype(np.int32)
    hkl = np.ascontiguousarray(hkl[(hkl ** 2).sum(1) <= r * r])
    cart = hkl * (2 * np.pi / n)
    return Basis(hkl=hkl, cart=cart, kpg=cart, kinetic=(cart ** 2).sum(1))


class _Box:
    """An n^3 box with a sphere of radius about n/4 and a random local potential."""

    def __init__(self, n, seed=0):
        self.grid = Grid(n, n, n, float(n ** 3))
        self.ctx = ApplyContext(self.grid, _sphere(n, n // 4), np.random.default_rng(seed).normal(size=n ** 3), [], [], self.grid.volume)


# FP64: the FFT's round-off, c eps log2(n^3) with c of order 10 against the largest entry: below 1e-13.
# FP32 passes: the same with the FP32 eps, below 5e-5 (the bounds of the smaller boxes' tests).
@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("path", ["planes", "sticks"])
def test_every_box_length(dz, monkeypatch, path, n):
    monkeypatch.delenv("DFTCUDA_FFT_PATH", raising=False)
    monkeypatch.setenv("DFTCUDA_LOCAL", path)
    box = _Box(n)
    x = random_block(box.ctx.n, 3, n)
    w = np.array([2.0, 0.5, 1.5])
    want, dens = box.ctx.apply_batch(x), odens.accumulate_density(box.grid, box.ctx.map, x, w, 1.0 / box.grid.volume)
    for prec, tol in ((0, 1e-13), (1, 5e-5)):
        if prec == 0 and n == 128:
            continue  # one FP64 plane of 128 x 128 does not fit shared memory: refused when the context is created
        kc = make_context(dz, box, precision=prec)
        assert rel_err(kc.apply_hamiltonian_batched(x), want) < tol
        assert kc.profile()["local_layout"] == (1 if path == "planes" else 2)
        rho = np.zeros(box.grid.count)
        kc.accumulate_band_density(x, w, rho)
        assert rel_err(rho, dens) < tol
        kc.close()


@pytest.mark.parametrize("weights", [[1.0], [0, 0, 2.0], [2.0, 1.0, 0, 0, 0], [0, 1.0, 2.0, 0.5, 0], [1.0, 0, 2.0, 0.5, 0, 0, 1.5], [0.0, -1.0]])
def test_density_of_scattered_bands(dz, weights):
    """Consecutive kept bands are read where they are; gaps, host memory and a start off the 16-byte
    boundary go through the staging copy.  The same bands in the same order: the same sums."""
    import torch

    kp = kproblem("si2", 20.0)
    kc = make_context(dz, kp)
    w = np.array(weights)
    v = random_block(kp.ctx.n, len(w), 8)
    v[w <= 0] = np.nan  # a band that is left out is not read
    ref = odens.accumulate_density(kp.grid, kp.ctx.map, v, w, 1.0 / kp.grid.volume)
    flat = torch.zeros(2 * v.size + 1, dtype=torch.float64, device="cuda")
    flat[1:] = torch.from_numpy(v.view(np.float64).ravel()).cuda()
    for vec in (v, torch.from_numpy(v).cuda(), flat[1:]):
        rho = torch.zeros(kp.grid.count, dtype=torch.float64, device="cuda")
        kc.accumulate_band_density(vec, w, rho)
        assert float((rho.cpu() - torch.from_numpy(ref)).abs().max()) <= 1e-12 * max(np.abs(ref).max(), 1.0)
    kc.close()


@pytest.mark.parametrize("axis", range(3))
@pytest.mark.parametrize("n", LENGTHS)
def test_fft_axis_lengths(dz, axis, n):
    """Each length along each axis, the other two leaving part of a block's lines unused."""
    dims = [5, 6, 3]
    dims[axis] = n
    x = random_block(int(np.prod(dims)), 1, n)[0]
    p = dz.Fft3dPlan(*dims)
    f, g = x.copy(), x.copy()
    p.forward(f)
    p.inverse(g)
    p.close()
    assert rel_err(f, offt.fft3d_forward(x, *dims)) < 1e-13
    assert rel_err(g, offt.fft3d_inverse(x, *dims)) < 1e-13


# one block's matrix ends at 95, the resident one of 148 SMs at 1205; a warp's lanes at 32 and 64
@pytest.mark.parametrize("m", [2, 31, 32, 33, 63, 65, 94, 95, 96, 97, 147, 149, 295, 297, 592, 593, 1184, 1185, 1205, 1206])
def test_subspace_sizes(dz, m):
    rng = np.random.default_rng(m)
    a = rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m))
    a = (a + a.conj().T) / 2
    nev = max(1, m // 3)
    r = dz.hermitian_eigen_decomp(a, nev)
    an = np.linalg.norm(a, 2)
    assert np.abs(r.values - np.linalg.eigvalsh(a)[:nev]).max() < 1e-12 * an
    res = np.linalg.norm(a @ r.vectors.T - r.vectors.T * r.values, axis=0)
    assert res.max() < 1e-12 * an * np.sqrt(m)
    assert np.abs(r.vectors.conj() @ r.vectors.T - np.eye(nev)).max() < 1e-10


@pytest.mark.parametrize("nbands", [1, 7, 8, 9, 31, 33, 92, 93, 100, 132])
def test_block_sizes_with_dropped_columns(dz, nbands):
    """Start vectors that repeat: the Gram matrix (the bands and a few more) loses the repeated ones, in one block up to
    96 columns and in panels of 32 above; the solve still reaches the dense eigenvalues."""
    kp = kproblem("si8", 12.0, (0.25, 0.0, 0.0))
    kc = make_context(dz, kp)
    x = random_block(kp.ctx.n, nbands, nbands)
    x[1::3] = x[: len(x[1::3])]
    r = kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, nbands, dz.Options(max_iter=300, tol=1e-8, init_vectors=x))
    kc.close()
    # a count that cuts a degenerate level need not reach the tolerance (the reference's restarts do not either): the
    # values' error is the residual's square over the gap (1e-10 / 1e-2), the vectors' orthonormality does not depend on it
    assert r.converged or r.max_residual < 1e-5
    assert np.abs(r.values - np.linalg.eigvalsh(kp.ctx.dense_hamiltonian())[:nbands]).max() < 1e-7
    assert np.abs(r.vectors.conj() @ r.vectors.T - np.eye(nbands)).max() < 1e-9


def test_resident_grids_of_concurrent_runs(dz):
    """Runs of one batch on their own streams, each with subspaces of 128 to 256: up to 128 blocks that each take an
    SM's shared memory, several grids wanting the chip at once.  The same eigenvalues as one at a time."""
    kps = [kproblem("si8", 12.0, (0.05 * i, 0.1, 0.0)) for i in range(6)]
    opts = dz.Options(max_iter=100, tol=1e-8)
    alone = []
    for kp in kps:
        kc = make_context(dz, kp)
        alone.append(kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, 64, opts).values)
        kc.close()
    kcs = [make_context(dz, kp) for kp in kps]
    both = dz.hermitian_eigen_decomp_iterative_batch(kcs, [kp.ctx.basis.kinetic for kp in kps], 64, opts)
    for kc in kcs:
        kc.close()
    for a, b in zip(alone, both):
        assert b.converged and np.abs(a - b.values).max() < 1e-9
