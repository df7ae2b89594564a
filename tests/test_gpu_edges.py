"""GPU kernels at the sizes where their tiles, splits and dispatch rules meet: tile edges
and remainders, odd leading dimensions and 8-byte aligned bases, the smallest and
largest orders of a rule, and both sides of each rule.

Tolerances, with u the unit roundoff of the type, derived from the operations:
  * triangular solves, backward and componentwise: each of at most m products and the
    64-wide inverted diagonal blocks adds a relative u of |T| |x|; the test matrices'
    blocks have |T_jj^-1| |T_jj| <= 4, so 4 (m + 64) u;
  * Cholesky |A - L L^T|_ij <= 4 (n + 64) u sqrt(a_ii a_jj), by the same count;
  * LU |P A - L U| <= 4 (min(m, n) + 64) u max(|L| |U|), pivots equal to LAPACK's;
  * products |C - C'| <= 2 (k + 4) u (|alpha| |A| |B| + |beta| |C|): both sides round.
"""
import threading

import numpy as np
import pytest
import scipy.linalg.lapack as la

from oracle import oracle as O

pytestmark = pytest.mark.gpu
U = np.finfo(np.float64).eps / 2
U32 = np.finfo(np.float32).eps / 2


@pytest.fixture(scope="module")
def lnb(cuda):
    import linompss_b200
    yield linompss_b200
    linompss_b200.set_chol_schedule(linompss_b200.SCHED_AUTO)
    linompss_b200.set_factor_mode(linompss_b200.FACTOR_TF32X3)


def dev(cuda, M, ld=None, off=0):
    """column-major device copy as a (cols, ld) view whose base lies `off` elements past an allocation; the
    rows past the matrix hold 7.25.  Returns (view, the whole buffer)"""
    import torch
    m, n = M.shape
    ld = ld or m
    host = np.full((n, ld), 7.25, dtype=M.dtype)
    host[:, :m] = M.T
    buf = torch.zeros(off + n * ld, dtype=torch.float64 if M.dtype == np.float64 else torch.float32, device=cuda)
    buf[off:] = torch.tensor(host.ravel(), device=cuda)
    return buf[off:].view(n, ld), buf


def tri(rng, m, uplo, diag):
    """well-conditioned triangle T, and T with NaN wherever it must not be read"""
    T = rng.standard_normal((m, m)) / np.sqrt(m) + 4 * np.eye(m)
    T = np.tril(T) if uplo == "L" else np.triu(T)
    Tn = T.copy()
    Tn[np.triu_indices(m, 1) if uplo == "L" else np.tril_indices(m, -1)] = np.nan
    if diag == "U":
        np.fill_diagonal(T, 1.0)
        np.fill_diagonal(Tn, np.nan)
    return T, Tn


# ---------------------------------------------------------------- triangular solves
def check_trsm(lnb, cuda, uplo, trans, diag, m, nrhs, alpha, pad, off):
    rng = np.random.default_rng(7 * m + nrhs)
    T, Tn = tri(rng, m, uplo, diag)
    B0 = rng.standard_normal((m, nrhs))
    Tt, _ = dev(cuda, Tn, m + pad, off)
    Bt, _ = dev(cuda, B0, m + pad, off)
    lnb.dtrsm_dev(uplo, trans, diag, m, nrhs, alpha, Tt, Bt)
    got = Bt.cpu().numpy()
    np.testing.assert_array_equal(got[:, m:], 7.25)
    X = got[:, :m].T
    op = T if trans == "N" else T.T
    bound = np.abs(op) @ np.abs(X) + abs(alpha) * np.abs(B0)
    assert (np.abs(op @ X - alpha * B0) / bound).max() <= 4 * (m + 64) * U


@pytest.mark.parametrize("uplo,trans,diag", [(a, b, c) for a in "LU" for b in "NT" for c in "NU"])
@pytest.mark.parametrize("m,nrhs,pad,off", [(1, 1, 0, 0), (63, 3, 1, 1), (64, 16, 0, 0), (65, 17, 0, 0),
                                            (129, 1, 2, 1), (200, 33, 3, 1), (577, 65, 0, 1)])
def test_trsm_forms(lnb, cuda, uplo, trans, diag, m, nrhs, pad, off):
    check_trsm(lnb, cuda, uplo, trans, diag, m, nrhs, 1.0 if nrhs % 2 else -2.5, pad, off)


@pytest.mark.parametrize("m,nrhs", [(1024, 512), (1024, 513), (2048, 2048), (2048, 2049), (4097, 1)])
def test_trsm_strip_widths(lnb, cuda, m, nrhs):
    """strips of 16, 32 and 64 columns by m x nrhs: both sides of each line"""
    check_trsm(lnb, cuda, "L", "N", "N", m, nrhs, 1.5, 0, 0)
    check_trsm(lnb, cuda, "L", "T", "U", m, nrhs, 1.0, 1, 1)


@pytest.mark.parametrize("n", [1, 31, 64, 65, 300])
@pytest.mark.parametrize("nrhs", [1, 9])
def test_spotrs_block_inverses(lnb, cuda, n, nrhs):
    """FP32 solves: the inverted blocks are computed in FP64 and held in FP32"""
    rng = np.random.default_rng(n + nrhs)
    L = tri(rng, n, "L", "N")[0].astype(np.float32)
    B0 = rng.standard_normal((n, nrhs)).astype(np.float32)
    Lt, _ = dev(cuda, L)
    Bt, _ = dev(cuda, B0)
    lnb.spotrs_dev(Lt, Bt, n, nrhs, "N")
    X = Bt.cpu().numpy().T.astype(np.float64)
    L64 = L.astype(np.float64)
    assert (np.abs(L64 @ X - B0) / (np.abs(L64) @ np.abs(X) + np.abs(B0))).max() <= 4 * (n + 64) * U32


# ---------------------------------------------------------------- Cholesky
def check_chol(A0, L, n, u=U, c=4):
    d = np.sqrt(np.diag(A0))
    L = np.tril(L).astype(np.float64)
    assert (np.abs(L @ L.T - A0) / np.outer(d, d)).max() <= c * (n + 64) * u


@pytest.mark.parametrize("sched", ["SCHED_DAG", "SCHED_STREAMS"])
@pytest.mark.parametrize("n,b,pad,off", [(1, 1, 0, 0), (31, 31, 0, 0), (33, 33, 2, 1), (64, 64, 0, 0), (65, 65, 1, 1),
                                         (127, 100, 0, 1), (129, 128, 1, 0), (191, 64, 0, 0), (193, 96, 0, 1),
                                         (257, 128, 2, 0), (449, 200, 1, 1), (1089, 250, 0, 1)])
def test_chol_edges(lnb, cuda, sched, n, b, pad, off):
    lnb.set_chol_schedule(getattr(lnb, sched))
    A0 = O.spd_covariance(n, 0.5, seed=n)
    A = np.tril(A0) + np.triu(np.full((n, n), np.nan), 1)      # the upper triangle is not read
    At, _ = dev(cuda, A, n + pad, off)
    lnb.dchol_dev(At, n, b)
    got = At.cpu().numpy()
    np.testing.assert_array_equal(got[:, n:], 7.25)
    assert np.isnan(got[:, :n].T[np.triu_indices(n, 1)]).all()
    check_chol(A0, np.tril(got[:, :n].T), n)


@pytest.mark.parametrize("sched,exp", [("SCHED_DAG", -1000), ("SCHED_DAG", -1060), ("SCHED_DAG", 1000),
                                       ("SCHED_STREAMS", -1000), ("SCHED_STREAMS", 1000)])
def test_chol_extreme_scale(lnb, sched, exp):
    """pivots near the ends of the exponent range: the factor is the unscaled one's, times 2^(exp/2).  (The streams'
    leaf forms 1 / pivot, which a subnormal pivot overflows: it reports that pivot.)"""
    lnb.set_chol_schedule(getattr(lnb, sched))
    n = 150
    A0 = O.spd_diag_dominant(n, seed=3)
    A = np.asfortranarray(np.ldexp(A0, exp))
    As = np.ldexp(A, -exp)                                      # what is left of the entries' bits
    assert lnb.ompss_dchol_rl(n, 64, 64, A, n) == 0
    L = np.ldexp(np.tril(A), -exp // 2)
    # at 2^-1060 the sums are subnormal: an absolute 2^-1074 each
    extra = (n + 64) * np.ldexp(1.0, -1074 - exp) if exp < -1022 else 0.0
    d = np.sqrt(np.diag(As))
    assert (np.abs(L @ L.T - As) - extra).max() <= 4 * (n + 64) * U * d.max() ** 2


@pytest.mark.parametrize("lo,hi", [(-1022, 1023), (-3, 3), (0, 0)])
def test_chol_reciprocal_root(lnb, cuda, lo, hi):
    """1/sqrt of a pivot d = 2^e m, e in [lo, hi]: [[d, 1], [1, c]] blocks leave 1 * (1/sqrt(d)) in L_21, exactly what
    the factor multiplies its columns by.  The walk's own iteration loses 1.5 u to its two roundings and 0.02 u to the
    series: at most 1.6 u off the exact value, and 3.6 u off CUDA's rsqrt (1 ulp, up to 2 u)."""
    import torch
    lnb.set_chol_schedule(lnb.SCHED_DAG)
    n, rng = 4096, np.random.default_rng(hi)
    for _ in range(3):
        d = np.ldexp(rng.uniform(1, 2, n // 2), rng.integers(lo, hi + 1, n // 2))
        d[:4] = np.ldexp([1.0, 1.0, 2 - 2.0 ** -52, 2 - 2.0 ** -52], [lo, hi, lo, hi])
        diag = np.empty(n)
        diag[::2] = d
        diag[1::2] = np.maximum(2 / d, 1.0)                     # the second pivot, c - 1/d, is normal and positive
        At = torch.diag(torch.tensor(diag, device=cuda))
        i = torch.arange(0, n, 2, device=cuda)
        At[i, i + 1] = 1.0                                      # column-major: A[i + 1, i]
        info = torch.full((1,), -9, dtype=torch.int32, device=cuda)
        lnb.dchol_dev(At, n, 256, info=info)
        assert int(info.item()) == 0
        got = At[i, i + 1].cpu().numpy()
        exact = 1 / np.sqrt(d.astype(np.longdouble))
        assert np.abs(got / exact - 1).max() <= 1.6 * U
        cuda_rsqrt = torch.rsqrt(torch.tensor(d, device=cuda)).cpu().numpy()
        assert np.abs(got / cuda_rsqrt.astype(np.longdouble) - 1).max() <= 3.6 * U
        root = At[i, i].cpu().numpy()                           # d * (1/sqrt(d)): one more rounding
        assert np.abs(root * exact - 1).max() <= 2.7 * U


@pytest.mark.parametrize("pos", [0, 6, 7, 15, 63, 71, 149])
def test_chol_infinite_pivot(lnb, pos):
    """1/sqrt(inf) = 0: the column below an infinite pivot is zero wherever it stands in its panel, so the rest of the
    factor is that of the matrix without this row and column"""
    lnb.set_chol_schedule(lnb.SCHED_DAG)
    n = 150
    A0 = O.spd_covariance(n, 0.5, seed=4)
    A = A0.copy(order="F")
    A[pos, pos] = np.inf
    assert lnb.ompss_dchol_rl(n, 64, 64, A, n) == 0
    L = np.tril(A)
    np.testing.assert_array_equal(L[pos + 1:, pos], 0.0)
    keep = np.arange(n) != pos
    check_chol(A0[np.ix_(keep, keep)], L[np.ix_(keep, keep)], n)


@pytest.mark.parametrize("sched", ["SCHED_DAG", "SCHED_STREAMS"])
@pytest.mark.parametrize("pos", [0, 1, 31, 32, 63, 64, 95, 127, 128, 199])
def test_chol_failed_pivot(lnb, sched, pos):
    """info names the pivot, the columns before its 32-column block are the factor's"""
    lnb.set_chol_schedule(getattr(lnb, sched))
    n = 200
    A0 = O.spd_covariance(n, 0.5, seed=11)
    L = np.linalg.cholesky(A0)
    A = A0.copy(order="F")
    A[pos, pos] = -1.0
    assert lnb.ompss_dchol_rl(n, 128, 128, A, n) == pos + 1
    k = pos // 64 * 64
    Ld = L.copy()
    Ld[pos, :] = np.where(np.arange(n) < pos, L[pos], Ld[pos])
    np.testing.assert_allclose(np.tril(A)[:k, :k], Ld[:k, :k], rtol=0, atol=64 * n * U * np.abs(L).max())


@pytest.mark.parametrize("n,b", [(1, 1), (31, 31), (33, 33), (64, 64), (97, 97), (127, 127), (128, 128), (500, 256),
                                 (600, 257), (700, 300), (1300, 513), (1700, 800), (1500, 999), (2300, 1023),
                                 (2100, 1024)])
@pytest.mark.parametrize("pad", [0, 1])
def test_schol_tiles(lnb, cuda, n, b, pad):
    """FP32 leaf and panel solves: narrow tiles, wide ones (257 to 1024 columns, the most a call takes), with
    and without 16-byte columns"""
    lnb.set_factor_mode(lnb.FACTOR_FP32)
    A0 = O.spd_covariance(n, 0.5, seed=n + b).astype(np.float32)
    At, _ = dev(cuda, A0, n + pad, pad)
    lnb.schol_dev(At, n, b)
    check_chol(A0.astype(np.float64), At.cpu().numpy()[:, :n].T, n, U32)


@pytest.mark.parametrize("pos", [0, 40, 127, 128, 700, 1029, 1299])
def test_schol_failed_pivot(lnb, pos):
    lnb.set_factor_mode(lnb.FACTOR_FP32)
    n, b = 1300, 640
    A = np.asfortranarray(O.spd_covariance(n, 0.5, seed=2).astype(np.float32))
    A[pos, pos] = -1.0
    assert lnb.ompss_schol_rl(n, b, b, A, n) == pos + 1


# ---------------------------------------------------------------- LU
def check_lu(A0, LU, ipiv):
    m, n = A0.shape
    k = min(m, n)
    perm = np.arange(m)
    for i, p in enumerate(ipiv):
        perm[[i, p - 1]] = perm[[p - 1, i]]
    L = np.tril(LU[:, :k], -1)
    L[np.arange(k), np.arange(k)] = 1.0
    Um = np.triu(LU[:k])
    assert np.abs(A0[perm] - L @ Um).max() <= 4 * (k + 64) * U * (np.abs(L) @ np.abs(Um)).max()


@pytest.mark.parametrize("m,n,pad,off", [(1, 1, 0, 0), (15, 17, 1, 1), (17, 15, 0, 1), (512, 40, 0, 0), (513, 40, 1, 1),
                                         (1024, 33, 0, 0), (1025, 33, 0, 1), (1536, 50, 0, 0), (1537, 50, 1, 0),
                                         (12288, 24, 0, 0), (12289, 24, 0, 1), (24576, 12, 0, 0), (24577, 12, 1, 0),
                                         (32768, 9, 0, 0), (2896, 2896, 0, 0), (2897, 2897, 1, 1), (700, 12000, 0, 0)])
def test_getrf_edges(lnb, cuda, m, n, pad, off):
    """panel shapes by rows (512, 1024, 1536 in one block, 12288 and 24576 by clusters), and the one-level and
    the blocked form (m n around 8 Mi)"""
    import torch
    A0 = np.random.default_rng(m + n).standard_normal((m, n))
    At, _ = dev(cuda, A0, m + pad, off)
    ipiv = torch.zeros(min(m, n), dtype=torch.int32, device=cuda)
    info = torch.full((1,), -9, dtype=torch.int32, device=cuda)
    lnb.dgetrf_dev(At, m, n, ipiv, info)
    got = At.cpu().numpy()
    assert int(info.item()) == 0
    np.testing.assert_array_equal(got[:, m:], 7.25)
    piv = ipiv.cpu().numpy()
    np.testing.assert_array_equal(piv, la.dgetrf(A0[:, :m])[1] + 1)      # the columns past m have no say
    check_lu(A0, got[:, :m].T, piv)


@pytest.mark.parametrize("rows", [512, 3000, 20000])
def test_getrf_multipliers(lnb, cuda, rows):
    """L's columns are the quotients a / pivot.  The panel forms them as a (1 / pivot) with the remainder put right
    (Markstein's theorem): the division's own bits, checked against numpy's division, wherever the remainder is exact
    (|a| >= 2^-968: its last bit is then at or above 2^-1074) and the quotient is normal; elsewhere within the last
    place.  Pivots on both sides of the range in which it does so, 1e-280 and 1e280."""
    import torch
    rng = np.random.default_rng(rows)
    tiny = np.finfo(np.float64).tiny
    for e in [0, 3, -700, 700, -929, -930, -931, 929, 930, 931, -1000, 1000, -1021, 1023]:
        pv = np.ldexp(rng.uniform(1, 2), e) * rng.choice([-1.0, 1.0])
        a = pv * rng.uniform(-1, 1, rows)
        a[1::2] = np.ldexp(a[1::2], rng.integers(-200, 1, a[1::2].size))
        a[3:6] = [0.0, np.nextafter(pv, 0), tiny * np.sign(pv)]
        a[7] = pv
        A0 = a[:, None].copy()
        At, _ = dev(cuda, A0)
        ipiv = torch.zeros(1, dtype=torch.int32, device=cuda)
        lnb.dgetrf_dev(At, rows, 1, ipiv)
        assert int(ipiv.item()) == 8
        got = At.cpu().numpy()[0]
        a[[0, 7]] = a[[7, 0]]
        with np.errstate(under="ignore"):
            q = a[1:] / pv
        assert got[0] == pv
        exact = (np.abs(a[1:]) >= 2.0 ** -968) & (np.abs(q) >= tiny) | (a[1:] == 0)
        np.testing.assert_array_equal(got[1:][exact], q[exact])
        assert (np.abs(got[1:] - q) <= np.spacing(np.abs(q))).all(), e


@pytest.mark.parametrize("n,nrhs,pad", [(1, 1, 0), (33, 1, 1), (1000, 3, 1), (1025, 17, 0), (1000, 40000, 0)])
def test_getrs_edges(lnb, cuda, n, nrhs, pad):
    """row exchanges of the right-hand sides, in one slice of scratch and in several (n nrhs > 32 Mi)"""
    import torch
    rng = np.random.default_rng(n + nrhs)
    A0 = rng.standard_normal((n, n)) + np.sqrt(n) * np.eye(n)[rng.permutation(n)]
    LU, piv, _ = la.dgetrf(A0)
    LUt, _ = dev(cuda, LU, n + pad)
    ipiv = torch.tensor(piv + 1, dtype=torch.int32, device=cuda)
    B0 = torch.randn(nrhs, n, dtype=torch.float64, device=cuda, generator=torch.Generator(cuda).manual_seed(n))
    Bt = torch.full((nrhs, n + pad), 7.25, dtype=torch.float64, device=cuda)
    Bt[:, :n] = B0
    lnb.dgetrs_dev(LUt, ipiv, Bt, n, nrhs)
    assert bool((Bt[:, n:] == 7.25).all())
    Aa = torch.tensor(A0, device=cuda)
    R = (Bt[:, :n] @ Aa.T - B0).abs()
    LUa = torch.tensor(np.abs(np.tril(LU, -1) + np.eye(n)) @ np.abs(np.triu(LU)), device=cuda)
    scale = LUa.sum(1).max() * Bt[:, :n].abs().max() + B0.abs().max()
    assert float(R.max() / scale) <= 12 * (n + 64) * U        # three such bounds: factor and two solves


@pytest.mark.parametrize("n,nrhs", [(1000, 3), (4096, 300), (1024, 8192)])
def test_getrs_after_a_timeout(lnb, cuda, n, nrhs):
    """a timeout that an earlier call left in the status word is not this call's (its waits look at that word once
    they have polled for a while: many columns)"""
    import ctypes
    import torch
    lib = lnb.lib()
    lib.lnb_selftest_wait_timeout.argtypes = [ctypes.c_longlong]
    g = torch.Generator(cuda).manual_seed(n)
    A = torch.randn(n, n, dtype=torch.float64, device=cuda, generator=g)
    A.diagonal().add_(2.0 * n)                                  # dominant: no growth, |L| |U| below 2 |A|
    At, piv = A.t().contiguous(), torch.zeros(n, dtype=torch.int32, device=cuda)
    lnb.dgetrf_dev(At, n, n, piv)
    B = torch.randn(nrhs, n, dtype=torch.float64, device=cuda, generator=g)
    Bt = B.clone()
    torch.cuda.synchronize()
    assert lib.lnb_selftest_wait_timeout(5000) == -5
    lnb.dgetrs_dev(At, piv, Bt, n, nrhs)
    scale = 2 * float(A.abs().sum(1).max() * Bt.abs().max()) + float(B.abs().max())
    assert float((Bt @ A.T - B).abs().max()) <= 12 * (n + 64) * U * scale


# ---------------------------------------------------------------- products
@pytest.mark.parametrize("ta,tb", [(a, b) for a in "NT" for b in "NT"])
@pytest.mark.parametrize("m,n,k,pad,off", [(1, 1, 1, 0, 0), (64, 64, 16, 0, 0), (65, 63, 17, 1, 1), (130, 70, 15, 0, 1),
                                           (128, 129, 33, 3, 0), (200, 1, 300, 0, 0), (1, 200, 31, 1, 1),
                                           (257, 255, 2, 0, 0)])
def test_gemm_edges(lnb, cuda, ta, tb, m, n, k, pad, off):
    rng = np.random.default_rng(m + n + k)
    A = rng.standard_normal((m, k) if ta == "N" else (k, m))
    B = rng.standard_normal((k, n) if tb == "N" else (n, k))
    Cm = rng.standard_normal((m, n))
    At, _ = dev(cuda, A, A.shape[0] + pad, off)
    Bt, _ = dev(cuda, B, B.shape[0] + pad, off)
    Ct, _ = dev(cuda, Cm, m + pad, off)
    lnb.dgemm_dev(ta, tb, m, n, k, -1.25, At, Bt, 0.75, Ct)
    got = Ct.cpu().numpy()
    np.testing.assert_array_equal(got[:, m:], 7.25)
    a, b = (A if ta == "N" else A.T), (B if tb == "N" else B.T)
    bound = 2 * (k + 4) * U * (1.25 * np.abs(a) @ np.abs(b) + 0.75 * np.abs(Cm))
    assert (np.abs(got[:, :m].T - (-1.25 * (a @ b) + 0.75 * Cm)) <= bound).all()


@pytest.mark.parametrize("uplo,trans", [(a, b) for a in "LU" for b in "NT"])
@pytest.mark.parametrize("n,k,pad,off", [(1, 1, 0, 0), (63, 17, 1, 1), (65, 64, 0, 0), (129, 15, 0, 1), (300, 130, 2, 0)])
def test_syrk_edges(lnb, cuda, uplo, trans, n, k, pad, off):
    rng = np.random.default_rng(n + k)
    A = rng.standard_normal((n, k) if trans == "N" else (k, n))
    Cm = rng.standard_normal((n, n))
    At, _ = dev(cuda, A, A.shape[0] + pad, off)
    Ct, _ = dev(cuda, Cm, n + pad, off)
    lnb.dsyrk_dev(uplo, trans, n, k, 0.5, At, -2.0, Ct)
    got = Ct.cpu().numpy()[:, :n].T
    a = A if trans == "N" else A.T
    keep = np.triu_indices(n, 1) if uplo == "L" else np.tril_indices(n, -1)
    np.testing.assert_array_equal(got[keep], Cm[keep])
    err = np.abs(got - (0.5 * a @ a.T - 2.0 * Cm))
    err[keep] = 0
    assert (err <= 2 * (k + 4) * U * (0.5 * np.abs(a) @ np.abs(a).T + 2 * np.abs(Cm))).all()


# the larger launch forms: K split over clusters of 8, 4 and 2 (few tiles, deep K), three CTAs per SM with the per-thread
# copy places (297 to 444 CTAs, alone and with K split; more than 592), the four-stage form between; odd leading
# dimensions, 8-byte bases and ragged K in each
@pytest.mark.parametrize("ta,tb", [(a, b) for a in "NT" for b in "NT"])
@pytest.mark.parametrize("m,n,k,pad,off", [(130, 70, 1040, 1, 1), (130, 70, 5035, 0, 0), (130, 130, 1001, 1, 0),
                                           (900, 800, 301, 1, 1), (900, 800, 300, 0, 0), (1281, 1025, 37, 1, 1),
                                           (1281, 1025, 50, 0, 0), (1500, 1300, 51, 1, 0), (1601, 1601, 131, 1, 1),
                                           (1602, 1601, 130, 0, 0), (1601, 1602, 15, 3, 0)])
def test_gemm_launch_forms(lnb, cuda, ta, tb, m, n, k, pad, off):
    import torch
    rng = np.random.default_rng(m + n + k)
    A = rng.standard_normal((m, k) if ta == "N" else (k, m))
    B = rng.standard_normal((k, n) if tb == "N" else (n, k))
    Cm = rng.standard_normal((m, n))
    At, _ = dev(cuda, A, A.shape[0] + pad, off)
    Bt, _ = dev(cuda, B, B.shape[0] + pad, off)
    Ct, _ = dev(cuda, Cm, m + pad, off)
    lnb.dgemm_dev(ta, tb, m, n, k, -1.25, At, Bt, 0.75, Ct)
    a, b, c = (torch.tensor(np.ascontiguousarray(x), device=cuda) for x in (A, B, Cm))
    a, b = (a if ta == "N" else a.T), (b if tb == "N" else b.T)
    bound = 2 * (k + 4) * U * (1.25 * a.abs() @ b.abs() + 0.75 * c.abs())
    assert bool((Ct[:, m:] == 7.25).all())
    assert bool(((Ct[:, :m].T - (-1.25 * (a @ b) + 0.75 * c)).abs() <= bound).all())


@pytest.mark.parametrize("uplo,trans", [(a, b) for a in "LU" for b in "NT"])
@pytest.mark.parametrize("n,k,pad,off", [(220, 5035, 1, 1), (220, 1008, 0, 0), (900, 401, 1, 0), (1200, 301, 1, 1),
                                         (1801, 37, 1, 1), (1800, 50, 0, 0), (2000, 51, 1, 0), (2301, 37, 1, 1),
                                         (2302, 130, 0, 0)])
def test_syrk_launch_forms(lnb, cuda, uplo, trans, n, k, pad, off):
    import torch
    rng = np.random.default_rng(n + k)
    A = rng.standard_normal((n, k) if trans == "N" else (k, n))
    Cm = rng.standard_normal((n, n))
    At, _ = dev(cuda, A, A.shape[0] + pad, off)
    Ct, _ = dev(cuda, Cm, n + pad, off)
    lnb.dsyrk_dev(uplo, trans, n, k, 0.5, At, -2.0, Ct)
    a, c = (torch.tensor(np.ascontiguousarray(x), device=cuda) for x in (A if trans == "N" else A.T, Cm))
    half = torch.tril if uplo == "L" else torch.triu
    got = Ct[:, :n].T
    assert bool((Ct[:, n:] == 7.25).all()) and torch.equal(got - half(got), c - half(c))
    bound = 2 * (k + 4) * U * (0.5 * a.abs() @ a.abs().T + 2 * c.abs())
    assert bool((half(got - (0.5 * a @ a.T - 2.0 * c)).abs() <= bound).all())


# one term per element, so the sum is exact up to its one rounding, and the last step is visible: beta C is not
# rounded before it joins alpha P.  m, n, k reach one CTA's form, K split over a cluster, and three CTAs per SM
@pytest.mark.parametrize("m,n,k", [(65, 63, 1), (200, 100, 2100), (1500, 1400, 3)])
@pytest.mark.parametrize("beta", [0.0, 0.7])
def test_gemm_epilogue_is_fused(lnb, cuda, m, n, k, beta):
    import torch
    from fractions import Fraction
    rng = np.random.default_rng(m)
    A, B = np.zeros((m, k)), np.zeros((k, n))
    A[:, k // 2], B[k // 2] = rng.standard_normal(m), rng.standard_normal(n)
    Cm = rng.standard_normal((m, n))
    alpha = 1.1
    (At, _), (Bt, _), (Ct, _) = dev(cuda, A), dev(cuda, B), dev(cuda, Cm)
    lnb.dgemm_dev("N", "N", m, n, k, alpha, At, Bt, beta, Ct)
    got = Ct.cpu().numpy().T
    for r, c in zip(rng.integers(0, m, 2000), rng.integers(0, n, 2000)):
        p = A[r, k // 2] * B[k // 2, c]
        assert got[r, c] == float(Fraction(alpha * p) + Fraction(beta) * Fraction(Cm[r, c])), (r, c)


def test_gemm_from_two_threads(lnb, cuda):
    """products use no workspace, so calls of several host threads may meet: neither may undo what the other's launch
    needs (the two orders here take different amounts of shared memory)"""
    import ctypes as C
    import torch
    errors, k = [], 8
    call = C.CDLL(lnb.LIB_PATH).lnb_dgemm_dev                  # the bare function: as little Python per call as can be

    def work(n):
        torch.cuda.set_device(cuda)
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            A, B = (torch.randn(n, k, dtype=torch.float64, device=cuda) for _ in range(2))
            Ct = torch.zeros(n, n, dtype=torch.float64, device=cuda)
        args = (C.c_char(b"T"), C.c_char(b"N"), C.c_int(n), C.c_int(n), C.c_int(k), C.c_double(1.0),
                C.c_void_p(A.data_ptr()), C.c_int(k), C.c_void_p(B.data_ptr()), C.c_int(k), C.c_double(0.0),
                C.c_void_p(Ct.data_ptr()), C.c_int(n), C.c_void_p(s.cuda_stream))
        rcs = set()
        for i in range(10000):
            rcs.add(call(*args))
            if i % 10 == 0:
                s.synchronize()
        s.synchronize()
        ok = bool(((Ct.T - A @ B.T).abs() <= 2 * (k + 4) * U * (A.abs() @ B.abs().T)).all())
        if rcs != {0} or not ok:
            errors.append((n, rcs, ok))

    threads = [threading.Thread(target=work, args=(n,)) for n in (500, 1000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


# ---------------------------------------------------------------- dense CG in one launch
@pytest.mark.parametrize("n,steps", [(1, 3), (2, 1), (31, 4), (33, 0), (64, 5), (1000, 6), (1501, 3)])
def test_dcg_edges(lnb, n, steps):
    """same steps as the oracle's loop.  A has a condition number below 4, so an error of 2 (n + 8) u per step
    grows by at most that per step"""
    A = np.asfortranarray(np.eye(n) * 3 + O.spd_covariance(n, 0.1, seed=n) / 4.2)
    rhs = np.random.default_rng(n).standard_normal(n)
    x = np.zeros(n)
    rc = lnb.ompss_dcg(n, 32, A, n, rhs.copy(), x, 1e-14, steps)
    rco, xo, _ = O.cg(A, rhs, 32, 1e-14, steps)
    assert rc == rco
    np.testing.assert_allclose(x, xo, rtol=0, atol=2 * (n + 8) * U * 4.0 ** max(steps, 1) * max(np.abs(xo).max(), 1e-300))


@pytest.mark.parametrize("n", [12288, 12289])
def test_dcg_largest_one_launch(lnb, n):
    """the largest order of the one-launch form, and the next; A = 3 I + a rank-one term, condition number below 4"""
    rng = np.random.default_rng(n)
    v = rng.uniform(-1, 1, n)
    A = np.empty((n, n), order="F")
    np.multiply.outer(v, v * (3.0 / n), out=A.T)               # symmetric in exact arithmetic; the upper triangle copied
    for r in range(0, n, 2048):
        A[r:, r:r + 2048] = A[r:r + 2048, r:].T.copy()
        B = A[r:r + 2048, r:r + 2048]
        B[:] = np.triu(B) + np.triu(B, 1).T
    A[np.arange(n), np.arange(n)] += 3
    rhs, x, steps = rng.standard_normal(n), np.zeros(n), 3
    rc = lnb.ompss_dcg(n, 512, A, n, rhs.copy(), x, 1e-14, steps)
    rco, xo, _ = O.cg(A, rhs, 512, 1e-14, steps)
    assert rc == rco
    np.testing.assert_allclose(x, xo, rtol=0, atol=2 * (n + 8) * U * 4.0 ** steps * np.abs(xo).max())


# ---------------------------------------------------------------- batched solves: both launch shapes
@pytest.mark.parametrize("extra", [0, 1])
@pytest.mark.parametrize("mode", ["FACTOR_FP32", "FACTOR_FP64"])
def test_batched_counts(lnb, cuda, mode, extra):
    """the two launch shapes meet at four systems per SM"""
    import torch
    count = 4 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    rng = np.random.default_rng(count)
    ns = rng.integers(1, 70, count)
    ns[:4] = [1, 512, 129, 256]
    rs = rng.integers(1, 9, count)
    As = [O.spd_covariance(int(n), 0.5, seed=i) for i, n in enumerate(ns)]
    Bs = [rng.standard_normal((n, r)) for n, r in zip(ns, rs)]
    ao = np.concatenate([[0], np.cumsum(ns.astype(np.int64) ** 2)])
    bo = np.concatenate([[0], np.cumsum(ns.astype(np.int64) * rs)])
    t = lambda v, d: torch.tensor(np.asarray(v), dtype=d, device=cuda)
    dA = t(np.concatenate([a.ravel(order="F") for a in As]), torch.float64)
    dB = t(np.concatenate([b.ravel(order="F") for b in Bs]), torch.float64)
    dX, info = torch.zeros_like(dB), torch.full((count,), -9, dtype=torch.int32, device=cuda)
    lnb.batched_posv_dev(t(ns, torch.int32), t(rs, torch.int32), t(ao[:-1], torch.int64), t(bo[:-1], torch.int64),
                         dA, dB, dX, getattr(lnb, mode), 10, info)
    assert (info.cpu().numpy() == 0).all()
    X = dX.cpu().numpy()
    for i, (A, B) in enumerate(zip(As, Bs)):
        n = int(ns[i])
        x = X[bo[i]:bo[i + 1]].reshape(B.shape, order="F")
        # refined to the FP64 level, or factored in FP64
        assert O.backward_error_np(A, x, B) <= 4 * (n + 64) * U, i


# ---------------------------------------------------------------- host matrices through the pinned slots
@pytest.mark.parametrize("n,lda", [(700, 700), (731, 731), (1537, 1600), (2001, 2001)])
def test_host_chol_large_copies(lnb, n, lda):
    """below and above the size from which copies are staged; the rest of the array is not written"""
    lnb.set_chol_schedule(lnb.SCHED_AUTO)
    A0 = O.spd_covariance(n, 0.5, seed=n)
    big = np.asfortranarray(np.full((lda, n), 7.25))
    big[:n] = A0
    assert lnb.ompss_dchol_rl(n, 256, 256, big, lda) == 0
    np.testing.assert_array_equal(big[n:], 7.25)
    np.testing.assert_array_equal(np.triu(big[:n], 1), np.triu(A0, 1))
    check_chol(A0, big[:n], n)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_host_lu_large_copies(lnb, dtype):
    A0 = np.random.default_rng(5).standard_normal((2503, 801)).astype(dtype)
    A = np.asfortranarray(A0.copy())
    info, ipiv = lnb.ompss_getrf(A, 801)
    assert info == 0
    L = np.tril(A, -1).astype(np.float64)
    L[np.arange(801), np.arange(801)] = 1.0
    Um = np.triu(A[:801]).astype(np.float64)
    perm = np.arange(2503)
    for i, p in enumerate(ipiv):
        perm[[i, p - 1]] = perm[[p - 1, i]]
    u = U if dtype == np.float64 else U32
    assert np.abs(A0[perm] - L @ Um).max() <= 4 * (801 + 64) * u * (np.abs(L) @ np.abs(Um)).max()


def test_host_calls_from_several_threads(lnb):
    """the pinned slots serve calls from any thread, one after another (calls at the same time share a workspace and
    are not offered); a release in between gives them back"""
    out = []

    def work(m):
        A0 = O.spd_covariance(m, 0.5, seed=m)
        B0 = O.fortran(np.random.default_rng(m).standard_normal((m, 3)))
        A, B = A0.copy(order="F"), B0.copy(order="F")
        out.append((lnb.dspdsolv_main(m, 3, 128, A, B), O.backward_error_np(A0, B, B0), m))

    for m in (900, 1201, 937):
        t = threading.Thread(target=work, args=(m,))
        t.start()
        t.join()
        if m == 1201:
            lnb.release_workspace()
    assert len(out) == 3
    for rc, berr, m in out:
        assert rc == 0 and berr <= 12 * (m + 64) * U


def test_host_copies_keep_the_callers_context(lnb):
    """A program with a CUDA context of its own (not the device's primary one): large pageable copies run in it, and it
    is current again, or rather still, after the call"""
    import os
    import subprocess
    import sys
    code = """
import ctypes as C, sys
import numpy as np
cu = C.CDLL("libcuda.so.1")
ctx, dev, now = C.c_void_p(), C.c_int(), C.c_void_p()
assert cu.cuInit(0) == 0 and cu.cuDeviceGet(C.byref(dev), 0) == 0
assert cu.cuCtxCreate_v2(C.byref(ctx), 0, dev) == 0
import linompss_b200 as lnb
m = 1100
T = np.asfortranarray(np.tril(np.random.default_rng(0).standard_normal((m, m))) / 30 + 4 * np.eye(m))
B0 = np.asfortranarray(np.random.default_rng(1).standard_normal((m, m)))
for _ in range(2):
    B = B0.copy(order="F")
    rc = lnb.ompss_dtrsm("L", "L", "N", "N", m, m, 64, 1.0, T, m, B, m)
    assert rc == 0, (rc, lnb.last_error())
    assert cu.cuCtxGetCurrent(C.byref(now)) == 0 and now.value == ctx.value, "another context is current"
    assert np.abs(T @ B - B0).max() <= 1e-11
print("same context")
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same context" in r.stdout, r.stdout + r.stderr
