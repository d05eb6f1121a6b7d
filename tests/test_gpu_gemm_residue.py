"""The FP64 complex GEMM's residue form (csrc/zgemm_i8.cu) at the edges of its tiles.

Entries are integers of at most 11 bits, so torch's complex128 product is exact and every difference is
the residue form's own.  Its entries are then exact too, which leaves the reconstruction (16 coefficients
cut at 76 bits for either part, times numbers below 2 p of moduli of sum 2736: 2^(12.5 - 76) P, P = 2^117.7, so 2^54.2
against scaled norms of at least 2^57 each: 2^-59 |a||b|) and four roundings of the result: 2^-58 |a||b| + 2^-51 |c| bounds both.  Where the
squares of a row leave the range its norm is bounded by sqrt(2 K) times the largest entry, up to 2^3.4
above the norm here: 2^-54 |a||b|."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ints(rows, k, kc, gen):
    x = torch.randint(-1024, 1025, (rows, k, 2), generator=gen, device=gen.device).double()
    x = torch.view_as_complex(x).cuda()
    return x if kc else x.T.contiguous().T


def _bound(a, b, ref, bits=58):
    na, nb = torch.linalg.vector_norm(a, dim=1), torch.linalg.vector_norm(b, dim=1)
    return 2.0 ** -bits * na[:, None] * nb[None, :] + 2.0 ** -51 * ref.abs()


def _assert_on_residues(dz, M, N, K, akc, bkc):
    """That products of this size run in the residue form: on random rows its error (2^-59 |a||b|) is below that of
    FP64 sums, which a corner of the same product takes, cut into up to 64 short sums (0.1 to 0.65 of it; the sums of the
    whole product are longer)."""
    rng = np.random.default_rng(M + N + K)
    a, b = (torch.randn((n, K) if kc else (K, n), dtype=torch.complex128, device="cuda", generator=torch.Generator("cuda").manual_seed(int(rng.integers(1 << 30))))
            for n, kc in ((M, akc), (N, bkc)))
    a, b = a if akc else a.T, b if bkc else b.T
    out, plain = dz.complex_gemm(a, b)[:32, :32].cpu().numpy(), dz.complex_gemm(a[:32], b[:32]).cpu().numpy()
    want = a[:32].cpu().numpy().astype(np.clongdouble) @ b[:32].cpu().numpy().astype(np.clongdouble).T
    err, err0 = (np.linalg.norm((x - want).astype(complex)) for x in (out, plain))
    assert err < 0.8 * err0, (err, err0)


# above the line of the size rule: rows around the 128- and 256-row tiles and the 8-row groups, columns around 32 and
# 256, K around the 64-deep blocks and the 128-deep slots; several K chunks, row chunks and output chunks
SHAPES = [(256, 256, 6016), (257, 255, 6017), (257, 513, 6001), (129, 1025, 2047), (1000, 97, 20000), (4000, 130, 1500), (513, 320, 16385),
          (700, 640, 1087), (2000, 224, 1056), (136, 300, 40000), (385, 289, 3073), (5000, 130, 8190), (600, 513, 60001), (1025, 1030, 33001),
          (131200, 520, 264)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("akc,bkc,cja,cjb", [(1, 1, 1, 0), (1, 0, 0, 0), (0, 0, 0, 1), (0, 1, 1, 1)])
def test_exact_on_integers(dz, M, N, K, akc, bkc, cja, cjb):
    _assert_on_residues(dz, M, N, K, akc, bkc)
    gen = torch.Generator("cuda").manual_seed(M + 3 * N + 7 * K)
    a, b = _ints(M, K, akc, gen), _ints(N, K, bkc, gen)
    o0 = torch.randint(-8, 9, (M, N), generator=gen, device="cuda").to(torch.complex128)
    ref = 2.0 * ((a.conj() if cja else a) @ (b.conj() if cjb else b).T) - o0
    for rowmajor in (True, False):
        out = o0.clone() if rowmajor else o0.T.contiguous().T
        dz.complex_gemm(a, b, out, conj_a=bool(cja), conj_b=bool(cjb), alpha=2.0, beta=-1.0)
        assert bool(((out - ref).abs() <= 2 * _bound(a, b, ref)).all()), (out - ref).abs().max().item()


def test_padded_strides(dz):
    _assert_on_residues(dz, 330, 300, 6000, 1, 0)
    gen = torch.Generator().manual_seed(5)
    a = _ints(330, 6100, True, gen)[:, 17:6017]
    b = _ints(6100, 310, False, gen)[50:6050].T[:300]
    out = torch.zeros(330, 640, dtype=torch.complex128, device="cuda")[:, 5:605:2]
    dz.complex_gemm(a, b, out)
    ref = a @ b.T
    assert bool(((out - ref).abs() <= _bound(a, b, ref)).all())


@pytest.mark.parametrize("shift", [0, -300, 300, -520, 480])
def test_rows_of_any_scale(dz, shift):
    """Rows scaled by powers of two far apart: every output is relative to its own rows' norms, also where
    their squares over- or underflow."""
    gen = torch.Generator().manual_seed(11)
    a, b = _ints(300, 2000, True, gen), _ints(400, 2000, True, gen)
    ref = a @ b.T
    bound = _bound(a, b, ref, 54 if abs(shift) > 400 else 58)
    # powers of two to the last bit (a device pow need not give them): the scaled entries stay exact
    sa = torch.from_numpy(np.ldexp(1.0, np.arange(300) % 40 + shift)).cuda()
    sb = torch.from_numpy(np.ldexp(1.0, -(np.arange(400) % 37))).cuda()
    out = dz.complex_gemm(a * sa[:, None], b * sb[:, None]) / sa[:, None] / sb[None, :]
    assert bool(((out - ref).abs() <= bound).all())


def test_zero_and_not_finite_rows(dz):
    gen = torch.Generator().manual_seed(12)
    a, b = _ints(300, 2000, True, gen), _ints(400, 2000, True, gen)
    ref = a @ b.T
    bound = _bound(a, b, ref)
    a[7], b[9] = 0, 0
    a[20, 5], a[21, 1999], b[33, 0] = complex(float("nan"), 0), complex(0, float("inf")), complex(float("-inf"), 1)
    out = dz.complex_gemm(a, b)
    rows, cols = torch.ones(300, dtype=torch.bool), torch.ones(400, dtype=torch.bool)
    rows[[20, 21]], cols[33] = False, False
    # infinities or NaN, as the FP64 sums give them
    assert not bool(torch.isfinite(out[[20, 21]]).any()) and not bool(torch.isfinite(out[:, 33]).any())
    assert float(out[7][cols.cuda()].abs().max()) == 0.0 and float(out[rows.cuda()][:, 9].abs().max()) == 0.0
    keep = rows.clone()
    keep[7] = False
    cols[9] = False
    assert bool(((out - ref).abs() <= bound)[keep.cuda()][:, cols.cuda()].all())


def test_without_room_for_the_tiles(dz):
    """When the tiles cannot be allocated the other FP64 kernel runs."""
    gen = torch.Generator().manual_seed(13)
    a, b = _ints(1400, 9000, True, gen), _ints(1400, 9000, True, gen)  # more room than any product above
    dz.debug_fail_alloc(0)
    try:
        out = dz.complex_gemm(a, b)
    except dz.OutOfMemory:  # the failure met the split-K workspace instead
        out = dz.complex_gemm(a, b)
    finally:
        dz.debug_fail_alloc()
    ref = a @ b.T
    assert float((out - ref).abs().max()) <= 1e-13 * float(ref.abs().max())


def test_not_less_exact_than_the_dmma_kernel(dz):
    """Against a double-double product: random columns (residues) are no further off than the FP64 tensor-core sums of eight
    columns of the product; band-like ones (uneven rows) keep FP64 sums, a few 2^-53 sqrt(K) of sum |a_k||b_k|."""
    rng = np.random.default_rng(3)
    K = 20000
    _assert_on_residues(dz, 160, 200, K, 1, 1)
    for envelope in (None, 1.0 / (1.0 + np.linspace(0, 25, K)) ** 1.5):
        a, b = (rng.normal(size=(n, K)) + 1j * rng.normal(size=(n, K)) for n in (160, 200))
        if envelope is not None:
            a, b = a * envelope, b * envelope
        want = (a.astype(np.clongdouble) @ b[:8].astype(np.clongdouble).T).astype(complex)
        out = dz.complex_gemm(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()).cpu().numpy()[:, :8]
        if envelope is None:
            plain = dz.complex_gemm(torch.from_numpy(a).cuda(), torch.from_numpy(b[:8]).cuda()).cpu().numpy()
            assert np.linalg.norm(out - want) <= 1.05 * np.linalg.norm(plain - want)
        else:
            assert (np.abs(out - want) <= 4 * K ** 0.5 * 2.0 ** -53 * (np.abs(a) @ np.abs(b[:8]).T)).all()


def test_projector_products_on_band_like_columns(dz):
    """A context's projector products take the residue form with whatever rows they have.  Its energies of 500 bands against
    those of 8 at a time (FP64 sums): the coefficients may differ by 2^-54 |P||x| of each, so E = 0.1 sum |c|^2 / Omega by
    2 * 2^-54 sqrt(rows) |P||x| |c| of 0.1 / Omega, with the largest row's |P|."""
    from tests.helpers import kproblem, make_context

    kp = kproblem("si8", 25.0, (0.25, 0.0, 0.0))
    kc = make_context(dz, kp)
    rng = np.random.default_rng(5)
    kin, n, rows = kp.ctx.basis.kinetic, kp.ctx.n, 5 * 512
    phi = rng.normal(size=(5, n)) * np.exp(-0.1 * kin)
    kc.set_projectors([dz.SpeciesProjectors([0, 0, 1], 0.1 * np.eye(3), phi)], np.zeros(512, dtype=np.int32), rng.uniform(0, 10.0, (512, 3)))
    size = np.linalg.norm(phi, axis=1).max()
    plain = (rng.normal(size=(500, n)) + 1j * rng.normal(size=(500, n)))
    steep = plain * np.exp(-0.4 * kin)
    spike = plain / (1.0 + kin) ** 1.5
    spike[:, np.argmax(kin)] *= 1e6
    for x in (plain, plain / (1.0 + kin) ** 1.5, steep, spike):
        got = kc.nonlocal_energies(x)
        want = np.concatenate([kc.nonlocal_energies(x[i : i + 8]) for i in range(0, 500, 8)])
        c = np.sqrt(want * kp.grid.volume / 0.1)
        bound = 0.1 / kp.grid.volume * 2 * 2.0 ** -54 * rows ** 0.5 * size * np.linalg.norm(x, axis=1) * c + 1e-14 * want
        assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()
    kc.close()


def test_many_k_splits(dz):
    """A product cut into 36 K splits, rows just above a power of two in norm (where the reconstruction's cut is largest
    against |a||b|).  Its coefficients lose less than 2^-76 each and multiply residues below p of 16 moduli of sum 2736:
    2^(11.5 - 76) P in either part, 2^-60.3 |a||b| for norms of at least 2^57 each, plus the roundings of the result."""
    gen = torch.Generator().manual_seed(14)
    a, b = (torch.view_as_complex(torch.randint(-728, 729, (160, 200000, 2), generator=gen).double()).cuda() for _ in range(2))
    ref = a @ b.T
    out = dz.complex_gemm(a, b)
    na, nb = torch.linalg.vector_norm(a, dim=1), torch.linalg.vector_norm(b, dim=1)
    assert bool(((out - ref).abs() <= 2.0 ** -60 * na[:, None] * nb[None, :] + 2.0 ** -51 * ref.abs()).all())


def _layout(x, kc):
    x = torch.from_numpy(x).cuda()
    return x if kc else x.T.contiguous().T


def _uneven(kind, rows, other, K, rng):
    """Pairs of operands whose large entries meet zeros or small entries of the other."""
    a, b = (rng.normal(size=(n, K)) + 1j * rng.normal(size=(n, K)) for n in (rows, other))
    if kind.startswith("outlier"):
        a[:, 1234] *= float(kind[7:])
        b[:, 1234] = 0
    elif kind == "one row":
        a[17, 77] *= 1e10
        b[:, 77] *= 1e-10
    elif kind == "halves":
        a[:, : K // 2] *= 1e-8
        b[:, K // 2 :] *= 1e-8
    elif kind == "sparse":
        a[:, ::2] = 0
        a[:, 1] *= 1e6
        b[:, 1::2] *= 1e-9
    return a, b


@pytest.mark.parametrize("kind", ["outlier1e8", "outlier1e12", "one row", "halves", "sparse"])
@pytest.mark.parametrize("akc,bkc", [(1, 1), (0, 1), (1, 0)])
def test_uneven_rows_keep_64_bit_sums(dz, kind, akc, bkc):
    """FP64 sums err by a few 2^-53 sqrt(K) of sum |a_k||b_k|, however far that is below |a||b|."""
    rng = np.random.default_rng(21)
    a, b = _uneven(kind, 300, 400, 4000, rng)
    out = dz.complex_gemm(_layout(a, akc), _layout(b, bkc)).cpu().numpy()
    at = np.s_[:20], np.s_[::50]
    want = (a[:20].astype(np.clongdouble) @ b[::50].astype(np.clongdouble).T).astype(complex)
    size = np.abs(a[:20]) @ np.abs(b[::50]).T
    assert (np.abs(out[at] - want) <= 4 * 4000 ** 0.5 * 2.0 ** -53 * size).all()
