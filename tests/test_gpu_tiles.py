"""Memory of the tensor-core products: the converted operands that contexts keep, and the workspaces."""
import numpy as np
import pytest
import torch

from tests.helpers import kproblem, make_context, random_block

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _set_projectors(dz, kp, kc, natoms, seed):
    rng = np.random.default_rng(seed)
    decay = np.exp(-0.1 * kp.ctx.basis.kinetic)
    kc.set_projectors([dz.SpeciesProjectors([0, 0, 1], 0.1 * np.eye(3), rng.normal(size=(5, kp.ctx.n)) * decay)],
                      np.zeros(natoms, dtype=np.int32), rng.uniform(0, 10.0, (natoms, 3)))


def _with_projectors(dz, natoms, precision=0, seed=3):
    """An 8-atom box whose projector matrix has 5 natoms rows: products of the residue form's size."""
    kp = kproblem("si8", 25.0, (0.25, 0.0, 0.0))
    kc = make_context(dz, kp, precision)
    _set_projectors(dz, kp, kc, natoms, seed)
    return kp, kc


def test_kept_tiles_give_way_on_a_full_device(dz):
    """One context keeps its projectors' tiles and its workspace; another one's solve needs more than what is left, but less
    than with the tiles freed: it runs, and the first context's results stay."""
    kp, kc = _with_projectors(dz, 512)
    x = torch.from_numpy(random_block(kp.ctx.n, 500, 7)).cuda()
    empty = _free()
    for _ in range(8):
        want = kc.apply_hamiltonian_batched(x, torch.empty_like(x)).clone()
    kept = empty - _free()
    kp2 = kproblem("si8", 20.0, (0.25, 0.0, 0.0))
    opts = dz.Options(max_iter=3, tol=1e-6)
    kin = kp2.ctx.basis.kinetic
    trial, late = make_context(dz, kp2), make_context(dz, kp2)
    before = _free()
    ref = trial.hermitian_eigen_decomp_iterative(kin, 60, opts)
    need = before - _free()
    trial.close()
    assert kept > 250 * MB and 30 * MB < need < kept
    filler = torch.empty(_free() - need // 2, dtype=torch.uint8, device="cuda")
    try:
        got = late.hermitian_eigen_decomp_iterative(kin, 60, opts)
    finally:
        del filler
        _free()
    assert np.abs(got.values - ref.values).max() < 1e-9
    again = kc.apply_hamiltonian_batched(x, torch.empty_like(x))
    assert float((again - want).abs().max()) <= 1e-13 * float(want.abs().max())
    late.close()
    kc.close()


def test_product_workspace_is_bounded(dz):
    """The residues of 4096 x 4096 outputs over 13 K chunks would take 7 GB: the outputs go in parts, and no more than 2 GB
    stay with the library after the call."""
    gen = torch.Generator(device="cuda").manual_seed(1)
    a, b = (torch.randn(4096, 100000, dtype=torch.complex128, device="cuda", generator=gen) for _ in range(2))
    small = torch.randn(64, 64, dtype=torch.complex128, device="cuda")
    dz.complex_gemm(small, small)
    before = _free()
    out = dz.complex_gemm(a, b)
    ref = torch.cat([a @ b[i : i + 512].T for i in range(0, 4096, 512)], 1)
    assert float(torch.linalg.vector_norm(out - ref)) < 1e-13 * float(torch.linalg.vector_norm(ref))
    del out, ref
    assert before - _free() <= 2100 * MB


@pytest.mark.parametrize("precision", [0, 1, 2, 3])
@pytest.mark.parametrize("sizes", [(2, 40), (300, 512), (512, 300), (512, 512)])
def test_projectors_set_anew_on_a_used_context(dz, precision, sizes):
    """More, fewer or as many projectors as before: every buffer follows, and what was kept of the old ones is not read."""
    cols = 500 if sizes[0] > 2 else 9
    kp, kc = _with_projectors(dz, sizes[0], precision)
    x = torch.from_numpy(random_block(kp.ctx.n, cols, 7)).cuda()
    y = torch.empty_like(x)
    for _ in range(12):
        kc.apply_hamiltonian_batched(x, y)
    _, fresh = _with_projectors(dz, sizes[1], precision, 4)
    _set_projectors(dz, kp, kc, sizes[1], 4)
    want = fresh.apply_hamiltonian_batched(x, torch.empty_like(x))
    tol = (1e-13, 5e-6, 5e-2, 2e-4)[precision]
    for _ in range(12):
        got = kc.apply_hamiltonian_batched(x, y)
        assert float((got - want).abs().max()) <= tol * float(want.abs().max())
    fresh.close()
    kc.close()


def test_first_products_keep_no_tiles(dz):
    """A context's first products convert the projectors in the workspace; the tiles of either product are kept, at different
    calls, once the conversions seen have cost what their buffers do.  Results do not depend on which it was."""
    kp, kc = _with_projectors(dz, 512)
    x = torch.from_numpy(random_block(kp.ctx.n, 500, 7)).cuda()
    y = torch.empty_like(x)
    want = kc.apply_hamiltonian_batched(x, y).clone()
    used = [-_free()]
    for _ in range(24):
        assert float((kc.apply_hamiltonian_batched(x, y) - want).abs().max()) <= 1e-13 * float(want.abs().max())
        used.append(-_free())
    tiles = 512 * 5 * kp.ctx.n * 32  # of one product
    grown = [b - a for a, b in zip(used, used[1:])]
    assert sum(g > tiles // 2 for g in grown) == 2 and not any(g > 1.5 * tiles for g in grown) and grown[0] < tiles // 2
    kc.close()


def test_contexts_of_several_threads_on_a_full_device(dz):
    """Two threads apply contexts that keep tiles while a third solves, again and again, on a context that needs what they
    keep: tiles go and come back under the running calls, and every result is as before."""
    import threading

    held = [_with_projectors(dz, 512, seed=s) for s in (3, 4)]
    n = held[0][0].ctx.n
    x = torch.from_numpy(random_block(n, 500, 7)).cuda()
    want = []
    for _, kc in held:
        for _ in range(8):
            y = kc.apply_hamiltonian_batched(x, torch.empty_like(x))
        want.append(y)
    kp = kproblem("si8", 20.0, (0.25, 0.0, 0.0))
    opts = dz.Options(max_iter=3, tol=1e-6)
    kcs = [make_context(dz, kp) for _ in range(6)]
    before = _free()
    ref = kcs[0].hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, 60, opts).values
    need = before - _free()
    out = [torch.empty_like(x) for _ in held]
    filler = torch.empty(_free() - need // 2, dtype=torch.uint8, device="cuda")
    errors = []

    def guarded(work, *args):
        try:
            work(*args)
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(repr(e))

    def apply(i):
        for _ in range(60):
            held[i][1].apply_hamiltonian_batched(x, out[i])
            bad = float((out[i] - want[i]).abs().max())
            assert bad <= 1e-13 * float(want[i].abs().max()), bad

    def solve():
        for kc in kcs[1:]:
            got = kc.hermitian_eigen_decomp_iterative(kp.ctx.basis.kinetic, 60, opts)
            assert np.abs(got.values - ref).max() < 1e-9
            kc.close()

    threads = [threading.Thread(target=guarded, args=a) for a in ((apply, 0), (apply, 1), (solve,))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    del filler
    for kc in [kcs[0]] + [h[1] for h in held]:
        kc.close()
    assert not errors, errors
