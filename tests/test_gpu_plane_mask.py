"""Tiles that hold one plane of the matrix only (real or imaginary): the kernels leave the other
plane out, and the results are those of the full complex product -- also for infinite and NaN
values, which the products left out would have spread to the other plane."""
import numpy as np
import pytest

from conftest import maxrel
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def planes(rows, cols, offsets, seed, scale=0.3):
    """Packed values whose 32-row tiles are, at random, zero, real, imaginary or complex."""
    rng = np.random.default_rng(seed)
    re, im = [], []
    for d in offsets:
        lo, L = max(0, -d), min(rows, cols - d) - max(0, -d)
        t = (lo + np.arange(L)) // 32
        kind = rng.integers(0, 4, (rows + 31) // 32)[t]
        re.append(np.where(kind & 1, rng.standard_normal(L) * scale, 0.0))
        im.append(np.where(kind & 2, rng.standard_normal(L) * scale, 0.0))
    return np.array(offsets, dtype=np.int32), np.concatenate(re), np.concatenate(im)


def full_product(rows, cols, off, re, im, X, tile=32):
    """A x row by row with all four products of every value in a tile of rows that holds a nonzero."""
    yr, yi = np.zeros((len(X), rows)), np.zeros((len(X), rows))
    p = 0
    with np.errstate(all="ignore"):
        for d in off:
            lo, L = max(0, -d), min(rows, cols - d) - max(0, -d)
            a, b, p = re[p:p + L], im[p:p + L], p + L
            t = (lo + np.arange(L)) // tile
            live = np.zeros((rows + tile - 1) // tile, dtype=bool)
            np.logical_or.at(live, t, (a != 0) | (b != 0))
            keep = live[t]
            r, a, b = (lo + np.arange(L))[keep], a[keep], b[keep]
            xr, xi = X.real[:, r + d], X.imag[:, r + d]
            yr[:, r] += a * xr
            yr[:, r] -= b * xi
            yi[:, r] += a * xi
            yi[:, r] += b * xr
    return yr, yi


def vectors(k, n, seed, special):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))
    if special:
        at = rng.choice(n, size=12, replace=False)
        for q in range(k):
            X.real[q, at[:3]] = [np.inf, np.nan, -np.inf]
            X.imag[q, at[3:6]] = [np.nan, np.inf, -np.inf]
            X[q, at[6]] = complex(np.inf, np.nan)
    return X


MANY = list(range(-140, 150))  # more than one chunk of staged metadata


@pytest.mark.parametrize("rows,cols,offs", [(3001, 2990, [0, 1, -1, 36, -37, 700, -701, 1501, 64]), (33, 40, [0, 2, -3]),
                                            (1100, 1100, MANY)])
@pytest.mark.parametrize("prec,k", [(0, 1), (0, 3), (1, 1), (1, 9)])
@pytest.mark.parametrize("special", [False, True])
def test_products_are_the_full_products(native, rows, cols, offs, prec, k, special):
    import torch

    capi, _ = native
    off, re, im = planes(rows, cols, offs, 7)
    dt = torch.float64 if prec != 1 else torch.float32
    if prec == 1:
        re, im = re.astype(np.float32).astype(float), im.astype(np.float32).astype(float)
    M = capi.Matrix.create(rows, cols, off, re, im, precision=prec)
    X = vectors(k, cols, 3, special)
    if prec == 1:
        X = X.astype(np.complex64).astype(complex)
    xr, xi = (torch.from_numpy(np.ascontiguousarray(v)).to("cuda", dt) for v in (X.real, X.imag))
    yr, yi = torch.empty(k, rows, device="cuda", dtype=dt), torch.empty(k, rows, device="cuda", dtype=dt)
    capi.check(capi.lib().diaq_spmm(M.h, k, xr.data_ptr(), xi.data_ptr(), cols, yr.data_ptr(), yi.data_ptr(), rows, None))
    want = full_product(rows, cols, off, re, im, X)
    tol = 1e-13 if prec == 0 else 1e-5  # sums of up to 290 products of order 1, in the vectors' precision
    for got, w in zip((yr, yi), want):
        got = got.double().cpu().numpy()
        assert np.array_equal(np.isnan(got), np.isnan(w))
        assert np.array_equal(got[np.isinf(w)], w[np.isinf(w)])
        ok = np.isfinite(w)
        assert maxrel(got[ok], w[ok]) < tol
        if special:
            assert not ok.all()


@pytest.mark.parametrize("rows,cols,offs", [(9001, 9005, [0, 1, -1, 36, -37, 700, -701, 1501, 64]), (70003, 70001, [0, 3, -64]),
                                            (270011, 270011, [0, -7, 1024])])
@pytest.mark.parametrize("prec,k", [(0, 1), (0, 3), (1, 1), (1, 5)])
@pytest.mark.parametrize("special", [False, True])
def test_larger_products_are_the_full_products(native, rows, cols, offs, prec, k, special):
    """The same through the kernels for more rows."""
    test_products_are_the_full_products(native, rows, cols, offs, prec, k, special)


@pytest.mark.parametrize("rows,cols,offs,k", [(208003, 208005, [0, 1, -1, 36, -37, 701, -207990, 208000], 5),
                                              (312007, 312001, [0, 3, -66, 1022], 3),
                                              (125004, 125004, [1, -3, 30, -1025, 2048], 9),
                                              (208005, 208011, MANY, 5)])
@pytest.mark.parametrize("special", [False, True])
def test_strip_products_are_the_full_products(native, rows, cols, offs, k, special):
    """3, 5 and 9 complex64 states at sizes where strips of 128 rows and 3 states take over: rows and
    columns off the tile sizes, diagonals of a few rows, more than one chunk of metadata, an incomplete
    chunk of states, aligned vectors with unaligned offsets."""
    test_products_are_the_full_products(native, rows, cols, offs, 1, k, special)


@pytest.mark.parametrize("rows", [70, 9001, 70003, 270011])
@pytest.mark.parametrize("prec,k", [(0, 1), (0, 3), (1, 1)])
def test_products_of_nan_vectors(native, rows, prec, k):
    """Sums that are NaN in both parts are not taken twice: vectors that hold NaN in both parts, in
    one, and infinities, in blocks (a product over several diagonals meets all mixtures)."""
    import torch

    capi, _ = native
    off, re, im = planes(rows, rows, [0, 1, -1, 33, -37], 17)
    dt = torch.float64 if prec != 1 else torch.float32
    if prec == 1:
        re, im = re.astype(np.float32).astype(float), im.astype(np.float32).astype(float)
    M = capi.Matrix.create(rows, rows, off, re, im, precision=prec)
    bad = np.array([complex(np.nan, np.nan), complex(np.nan, 1), complex(2, np.nan), complex(np.inf, 1), complex(1, -np.inf), 1 + 1j])
    rng = np.random.default_rng(8)
    X = bad[np.repeat(np.minimum(rng.integers(0, 15, (k, rows // 23 + 1)), 5), 23, axis=1)[:, :rows]]
    xr, xi = (torch.from_numpy(np.ascontiguousarray(v)).to("cuda", dt) for v in (X.real, X.imag))
    yr, yi = torch.empty(k, rows, device="cuda", dtype=dt), torch.empty(k, rows, device="cuda", dtype=dt)
    capi.check(capi.lib().diaq_spmm(M.h, k, xr.data_ptr(), xi.data_ptr(), rows, yr.data_ptr(), yi.data_ptr(), rows, None))
    for got, w in zip((yr, yi), full_product(rows, rows, off, re, im, X)):
        got = got.double().cpu().numpy()
        assert np.array_equal(np.isnan(got), np.isnan(w))
        assert np.array_equal(got[np.isinf(w)], w[np.isinf(w)])
        ok = np.isfinite(w)
        assert ok.any() and maxrel(got[ok], w[ok]) < (1e-13 if prec == 0 else 1e-5)


def _evolve(capi, H, N, X, mode, cfg):
    import torch

    E = capi.Evolve(H, len(X), mode)
    E.set_config(*cfg)
    pr, pi = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (X.real, X.imag))
    E.run(pr, pi, N, 0.05, 1, 0, 3)
    return np.stack([pr.cpu().numpy(), pi.cpu().numpy()])


@pytest.mark.parametrize("k", [1, 4, 9])
@pytest.mark.parametrize("mode", ["c128", "mixed", "horner"])
def test_plans_are_the_full_products(native, k, mode):
    """The plan kernels that look at the planes against the ones that always take both (the c128
    plan: against the oracle), also with infinite and NaN states."""
    capi, _ = native
    N = 2100
    off, re, im = planes(N, N, [0, 1, -1, 37, -37, 700, -700, 64, 5], 9)
    H = capi.Matrix.create(N, N, off, re, im)
    X = vectors(k, N, 4, False)
    X /= np.linalg.norm(X, axis=1, keepdims=True)
    bad = vectors(k, N, 4, True)
    if mode == "c128":
        A = orc.OMatrix(N, N, off, re, im)
        for cfg in ((8, 1, 0), (4, 2, 0), (1, 2, 0)):
            got = _evolve(capi, H, N, X, capi.EVOLVE_C128, cfg)
            for q in range(k):
                assert maxrel(got[0, q] + 1j * got[1, q], orc.ham_sim(A, X[q], 0.05, 1, 3)) < 1e-12
        return
    md = capi.EVOLVE_MIXED if mode == "mixed" else capi.EVOLVE_HORNER
    for P in (X, bad):
        want = _evolve(capi, H, N, P, md, (4, 1, 9))
        assert np.isfinite(want).all() == (P is X)
        for cfg in ((8, 1, 0), (4, 2, 0), (8, 4, 0), (4, 1, 12)):
            got = _evolve(capi, H, N, P, md, cfg)
            assert np.array_equal(got, want, equal_nan=True), cfg


def _special(off, rows, cols, re, im, seed):
    """The matrix with every tile holding a nonzero, and a few infinite and NaN values."""
    rng = np.random.default_rng(seed)
    p = 0
    for d in off:
        L = min(rows, cols - d) - max(0, -d)
        t = (max(0, -d) + np.arange(L)) // 32
        live = np.zeros((rows + 31) // 32, dtype=bool)
        np.logical_or.at(live, t, (re[p:p + L] != 0) | (im[p:p + L] != 0))
        re[p:p + L][~live[t]] = 0.25
        p += L
    at = rng.choice(len(re), size=6, replace=False)
    re[at[:2]], im[at[2:4]] = [np.inf, np.nan], [np.nan, -np.inf]
    return re, im


@pytest.mark.parametrize("prec,tol", [(0, 1e-13), (1, 1e-5)])
@pytest.mark.parametrize("rows,inner,cols,offa,offb", [(1030, 1001, 1100, [0, 1, -3, 33, -65, 200], [0, -1, 5, 31, -40, 130]),
                                                       (70, 64, 33, [0, -37, 2], [0, 1, -1]),
                                                       (300, 300, 300, list(range(-45, 45)), list(range(-50, 50)))])
@pytest.mark.parametrize("special", [False, True])
def test_matrix_products_are_the_full_products(native, prec, tol, rows, inner, cols, offa, offb, special):
    """A B by planes: more pairs per result diagonal than a warp stages at once (the third shape),
    odd offsets, rectangular shapes; sums of at most 90 products of order 0.1."""
    import ctypes

    capi, _ = native
    oa, ra, ia = planes(rows, inner, offa, 11)
    ob, rb, ib = planes(inner, cols, offb, 12)
    if special:
        ra, ia = _special(oa, rows, inner, ra, ia, 5)
        rb, ib = _special(ob, inner, cols, rb, ib, 6)
    if prec == 1:
        ra, ia, rb, ib = (v.astype(np.float32).astype(float) for v in (ra, ia, rb, ib))
    A = capi.Matrix.create(rows, inner, oa, ra, ia, precision=prec)
    B = capi.Matrix.create(inner, cols, ob, rb, ib, precision=prec)
    out = ctypes.c_void_p()
    capi.check(capi.lib().diaq_spgemm(A.h, B.h, 0, None, ctypes.byref(out)))
    off, re, im = capi.Matrix(out).download()
    want = {}
    pa = 0
    with np.errstate(all="ignore"):
        for da in oa:
            lo, L = max(0, -da), min(rows, inner - da) - max(0, -da)
            a, b, pa = ra[pa:pa + L], ia[pa:pa + L], pa + L
            pb = 0
            for db in ob:
                lob, Lb = max(0, -db), min(inner, cols - db) - max(0, -db)
                c, d, pb = rb[pb:pb + Lb], ib[pb:pb + Lb], pb + Lb
                r0, r1 = max(lo, lob - da), min(lo + L, lob + Lb - da)
                if r0 >= r1:
                    continue
                wr, wi = want.setdefault(da + db, (np.zeros(rows), np.zeros(rows)))
                u, v, x, y = a[r0 - lo:r1 - lo], b[r0 - lo:r1 - lo], c[r0 + da - lob:r1 + da - lob], d[r0 + da - lob:r1 + da - lob]
                wr[r0:r1] += u * x
                wr[r0:r1] -= v * y
                wi[r0:r1] += u * y
                wi[r0:r1] += v * x
    assert set(want) <= set(off.tolist())
    p = 0
    bad = 0
    for dc in off.tolist():
        lo, L = max(0, -dc), min(rows, cols - dc) - max(0, -dc)
        for got, w in ((re, want.get(dc, (np.zeros(rows),) * 2)[0]), (im, want.get(dc, (np.zeros(rows),) * 2)[1])):
            g, w = got[p:p + L], w[lo:lo + L]
            assert np.array_equal(np.isnan(g), np.isnan(w)), dc
            assert np.array_equal(g[np.isinf(w)], w[np.isinf(w)]), dc
            ok = np.isfinite(w)
            bad += int((~ok).sum())
            assert np.abs(g[ok] - w[ok]).max(initial=0.0) < tol * 10, dc
        p += L
    assert (bad > 0) == special


@pytest.mark.parametrize("offs", [[0, 1, -1, 37, -37, 700, 64, 5], list(range(-130, 140))])
@pytest.mark.parametrize("k", [4, 9])
@pytest.mark.parametrize("mode", ["mixed", "horner"])
@pytest.mark.parametrize("special", [False, True])
def test_real_matrices_in_the_interleaved_kernels(native, offs, k, mode, special):
    """A matrix without an imaginary part: the interleaved plan kernel and the interleaved batched
    kernel give the bits of the kernels that take both planes, also for infinite and NaN states."""
    import torch

    capi, _ = native
    N = 1500
    off, re, im = planes(N, N, offs, 21, scale=0.05)
    im[:] = 0
    H = capi.Matrix.create(N, N, off, re, im)
    X = vectors(k, N, 5, special) * 0.1
    md = capi.EVOLVE_MIXED if mode == "mixed" else capi.EVOLVE_HORNER
    want = _evolve(capi, H, N, X, md, (4, 1, 9))
    assert np.isfinite(want).all() != special
    assert np.array_equal(_evolve(capi, H, N, X, md, (4, 1, 12)), want, equal_nan=True)
    got = []
    for il in (True, False):
        pr, pi = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (X.real, X.imag))
        B = capi.Batch([H.convert(capi.C64)], [pr], [pi])
        B.set_horner(mode == "horner")
        B.set_interleaved(il)
        B.set_config(4, 1)
        B.run(0.05, [0], [3], 1)
        torch.cuda.synchronize()
        got.append(np.stack([pr.cpu().numpy(), pi.cpu().numpy()]))
    assert np.array_equal(got[0], got[1], equal_nan=True)
    assert np.array_equal(got[0], want, equal_nan=True)


@pytest.mark.parametrize("rows,cols,offs,real", [(3001, 2990, [0, 1, -1, 36, -37, 700, -701, 1501, 64], False),
                                                 (1100, 1100, MANY, False), (33, 40, [0, 2, -3], True),
                                                 (800003, 800001, [0, 3, -70001], True),
                                                 (800003, 800001, [0, 3, -70001], False)])
@pytest.mark.parametrize("k", [1, 3])
@pytest.mark.parametrize("special", [False, True])
def test_float_pair_products_are_the_full_products(native, rows, cols, offs, real, k, special):
    """Float pairs, both kernels, one and three states: the values, and non-finite results where the
    full product has them (TwoSum turns an infinity into NaN).  The kernel with four rows per thread
    takes a zero tile along when its strip of 128 rows is live and the offset is not a multiple of 4:
    0 * infinity may show in such a strip, and nowhere else."""
    import torch

    capi, _ = native
    off, re, im = planes(rows, cols, offs, 13)
    if real:
        im[:] = 0
    M = capi.Matrix.create(rows, cols, off, re, im, precision=capi.C128F2)
    X = vectors(k, cols, 3, special)
    xr, xi = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (X.real, X.imag))
    yr, yi = torch.empty(k, rows, device="cuda", dtype=torch.float64), torch.empty(k, rows, device="cuda", dtype=torch.float64)
    capi.check(capi.lib().diaq_spmm(M.h, k, xr.data_ptr(), xi.data_ptr(), cols, yr.data_ptr(), yi.data_ptr(), rows, None))
    strips = full_product(rows, cols, off, re, im, X, tile=128)
    for got, w, ws in zip((yr, yi), full_product(rows, cols, off, re, im, X), strips):
        got = got.cpu().numpy()
        assert not np.isfinite(got[~np.isfinite(w)]).any()
        assert np.isfinite(got[np.isfinite(ws)]).all()
        ok = np.isfinite(ws)
        assert maxrel(got[ok], w[ok]) < 1e-12   # 2^-48 per value, up to 290 of them
        assert ok.all() != special
