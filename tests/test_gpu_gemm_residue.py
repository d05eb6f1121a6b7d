"""The FP64 complex GEMM's residue form (csrc/zgemm_i8.cu) at the edges of its tiles.

Entries are integers of at most 11 bits, so torch's complex128 product is exact and every difference is
the residue form's own.  Its entries are then exact too, which leaves the reconstruction (32 coefficients
cut at 76 bits times residue sums below 2^9 P, P = 2^117.7: 2^54.6 against scaled norms of at least 2^57
each, so 2^-59 |a||b|) and four roundings of the result: 2^-58 |a||b| + 2^-51 |c| bounds both.  Where the
squares of a row leave the range its norm is bounded by sqrt(2 K) times the largest entry, up to 2^3.4
above the norm here: 2^-54 |a||b|."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ints(rows, k, kc, gen):
    x = torch.randint(-1024, 1025, (rows, k, 2), generator=gen).double()
    x = torch.view_as_complex(x).cuda()
    return x if kc else x.T.contiguous().T


def _bound(a, b, ref, bits=58):
    na, nb = torch.linalg.vector_norm(a, dim=1), torch.linalg.vector_norm(b, dim=1)
    return 2.0 ** -bits * na[:, None] * nb[None, :] + 2.0 ** -51 * ref.abs()


# rows around the 128- and 256-row tiles and the 8-row groups, columns around 32 and 256, K around the
# 64-deep blocks, the 128-deep slots and the K chunks
SHAPES = [(256, 256, 3008), (257, 255, 3009), (129, 1025, 2047), (32, 4000, 1500), (513, 33, 16385), (700, 320, 1087), (2000, 96, 1056),
          (40, 140, 40000), (131200, 33, 264)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("akc,bkc,cja,cjb", [(1, 1, 1, 0), (1, 0, 0, 0), (0, 0, 0, 1), (0, 1, 1, 1)])
def test_exact_on_integers(dz, M, N, K, akc, bkc, cja, cjb):
    gen = torch.Generator().manual_seed(M + 3 * N + 7 * K)
    a, b = _ints(M, K, akc, gen), _ints(N, K, bkc, gen)
    o0 = torch.randint(-8, 9, (M, N), generator=gen).to(torch.complex128).cuda()
    ref = 2.0 * ((a.conj() if cja else a) @ (b.conj() if cjb else b).T) - o0
    for rowmajor in (True, False):
        out = o0.clone() if rowmajor else o0.T.contiguous().T
        dz.complex_gemm(a, b, out, conj_a=bool(cja), conj_b=bool(cjb), alpha=2.0, beta=-1.0)
        assert bool(((out - ref).abs() <= 2 * _bound(a, b, ref)).all()), (out - ref).abs().max().item()


def test_padded_strides(dz):
    gen = torch.Generator().manual_seed(5)
    a = _ints(330, 2100, True, gen)[:, 17:2017]
    b = _ints(2100, 310, False, gen)[50:2050].T[:300]
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
    """Against a double-double product, on band-like columns and on random ones: no further off than the
    FP64 tensor-core sums of the same product."""
    rng = np.random.default_rng(3)
    K = 20000
    for envelope in (np.ones(K), 1.0 / (1.0 + np.linspace(0, 25, K)) ** 1.5):
        a = (rng.normal(size=(64, K)) + 1j * rng.normal(size=(64, K))) * envelope
        b = (rng.normal(size=(160, K)) + 1j * rng.normal(size=(160, K))) * envelope
        want = a.astype(np.clongdouble) @ b[:8].astype(np.clongdouble).T
        out = dz.complex_gemm(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()).cpu().numpy()[:, :8]
        plain = dz.complex_gemm(torch.from_numpy(a[:, :]).cuda(), torch.from_numpy(b[:8]).cuda()).cpu().numpy()  # 8 columns: the DMMA kernel
        err, err0 = (np.linalg.norm((x - want).astype(complex)) for x in (out, plain))
        assert err <= 1.05 * err0, (err, err0)


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


@pytest.mark.parametrize("akc,bkc", [(1, 1), (0, 0)])
@pytest.mark.parametrize("M,N,K", [(300, 400, 4000), (129, 1025, 2047), (330, 300, 6007)])
def test_even_rows_run_on_residues(dz, M, N, K, akc, bkc):
    """Random rows stay in the residue form, whose error (2^-59 |a||b|) is far below the FP64 sums'."""
    rng = np.random.default_rng(22)
    a, b = (rng.normal(size=(n, K)) + 1j * rng.normal(size=(n, K)) for n in (M, N))
    da, db = _layout(a, akc), _layout(b, bkc)
    out = dz.complex_gemm(da, db).cpu().numpy()[:, :8]
    plain = dz.complex_gemm(da, db[:8]).cpu().numpy()  # too few columns: the FP64 kernel
    want = a.astype(np.clongdouble) @ b[:8].astype(np.clongdouble).T
    err, err0 = (np.linalg.norm((x - want).astype(complex)) for x in (out, plain))
    assert err < 0.5 * err0, (err, err0)
