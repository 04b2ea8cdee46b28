"""Block products whose fragments are read straight from global memory
(pb_frag.cuh): odd widths and offsets, partial 8-column tiles, row counts
around a chunk's end, W'W, in-place updates; columns beside the views hold
NaN and must not reach a result.

Bound: sums of n products, componentwise against t = |V|'|W|: n eps t in FP64;
FP32 results are formed in FP64 and rounded once, so n eps64 t plus one eps of
the result, except in the wide aligned products, which a staged kernel sums in
FP32: there no chain of additions is longer than the 32 to 256 rows of a tile
plus 157 blocks, 512 in all.  A dropped or doubled row moves an entry by its
product, some 1/4, which is above these bounds.  The row-local products add at
most m + 3 roundings of numbers of at most m + 3."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _block(n, ld, off, w, rng, dtype):
    """an n x w view at column off of a block of ld columns, NaN around it"""
    from phist_b200.objects import Map, Mvec
    a = np.full((n, ld), np.nan, dtype)
    a[:, off:off + w] = rng.uniform(-1, 1, (n, w)).astype(dtype)
    mp = Map(n)
    b = Mvec(mp.h, ld, dtype).set(a)
    return mp, b, b.view(off, off + w - 1), a[:, off:off + w].astype(np.float64)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m,k,vo,vld,wo,wld", [
    (5, 1, 0, 5, 0, 1), (8, 5, 1, 10, 3, 9), (9, 7, 0, 10, 1, 8), (10, 4, 0, 10, 0, 4), (17, 9, 2, 20, 0, 10),
    (37, 5, 0, 47, 0, 5), (40, 8, 0, 40, 0, 8), (24, 16, 0, 24, 0, 16), (5, 41, 1, 6, 0, 41), (33, 33, 1, 35, 1, 34),
    (64, 64, 1, 66, 1, 66), (64, 20, 0, 64, 0, 20)])
@pytest.mark.parametrize("n", [1, 31, 160, 161, 5003])
def test_products(session, n, m, k, vo, vld, wo, wld, dtype):
    from phist_b200 import kernels as K
    from phist_b200.objects import SdMat, fn
    rng = np.random.default_rng(n + 100 * m + k)
    mp, Vb, V, v = _block(n, vld, vo, m, rng, dtype)
    mq, Wb, W, w = _block(n, wld, wo, k, rng, dtype)
    eps = np.finfo(dtype).eps
    c0 = rng.uniform(-1, 1, (m, k)).astype(dtype)
    C = SdMat(m, k, dtype).set(c0)
    K.chk(fn(dtype, "mvecT_times_mvec"), 0.5, V.h, W.h, 2.0, C.h)
    ref = 0.5 * (v.T @ w) + 2.0 * c0
    e64 = np.finfo(np.float64).eps
    terms = 0.5 * (np.abs(v).T @ np.abs(w)) + 2.0 * np.abs(c0)
    staged = dtype == np.float32 and (m, k, vo, wo) in ((24, 16, 0, 0), (64, 20, 0, 0))
    assert (np.abs(C.get() - ref) <= ((n + 3) * e64 + (512 if staged else 1) * eps) * terms).all()
    G = SdMat(k, k, dtype)
    K.chk(fn(dtype, "mvecT_times_mvec"), 1.0, W.h, W.h, 0.0, G.h)
    g = G.get()
    assert (np.abs(g - w.T @ w) <= ((n + 3) * e64 + eps) * (np.abs(w).T @ np.abs(w))).all()
    if k <= 32:
        assert np.array_equal(g, g.T)
    C.set(c0)
    K.chk(fn(dtype, "mvec_times_sdMat"), -0.5, V.h, C.h, 2.0, W.h)
    ref = -0.5 * (v @ c0.astype(np.float64)) + 2.0 * w
    got = Wb.get()
    assert np.abs(got[:, wo:wo + k] - ref).max() <= (m + 3) * (m + 3) * eps
    beside = np.delete(got, np.s_[wo:wo + k], axis=1)
    assert np.isnan(beside).all()
    if k <= m:
        K.chk(fn(dtype, "mvec_times_sdMat_inplace"), V.h, C.h)
        got = Vb.get()[:, vo:vo + m]
        assert np.abs(got[:, :k] - v @ c0.astype(np.float64)).max() <= (m + 3) * (m + 3) * eps
        assert np.array_equal(got[:, k:], v[:, k:].astype(dtype))
    for o in (V, W, C, G, Vb, Wb, mp, mq):
        o.delete()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m,k", [(2, 3), (5, 4), (16, 16), (20, 17), (33, 33), (48, 8), (64, 64)])
def test_no_rows(session, m, k, dtype):
    """blocks without rows: the sum is empty, C = beta C"""
    from phist_b200 import kernels as K
    from phist_b200.objects import Map, Mvec, SdMat, fn
    mp = Map(0)
    V, W = Mvec(mp.h, m, dtype), Mvec(mp.h, k, dtype)
    c0 = np.arange(m * k, dtype=dtype).reshape(m, k)
    C = SdMat(m, k, dtype).set(c0)
    K.chk(fn(dtype, "mvecT_times_mvec"), 1.0, V.h, W.h, 2.0, C.h)
    assert np.array_equal(C.get(), 2 * c0)
    K.chk(fn(dtype, "mvec_times_sdMat"), 1.0, V.h, C.h, 2.0, W.h)
    for o in (V, W, C, mp):
        o.delete()


def test_infinity_stays_in_its_row(session):
    """an infinite entry in the last column meets no zero padding"""
    from phist_b200 import kernels as K
    from phist_b200.objects import SdMat
    rng = np.random.default_rng(3)
    n, m, k = 100, 13, 6
    mp, Vb, V, v = _block(n, m, 0, m, rng, np.float64)
    v[7, m - 1] = np.inf
    Vb.set(v)
    mq, Wb, W, w = _block(n, k, 0, k, rng, np.float64)
    C = SdMat(m, k).set(np.ones((m, k)))
    K.chk(K.phist_Dmvec_times_sdMat, 1.0, V.h, C.h, 0.0, W.h)
    got = Wb.get()
    assert np.isposinf(got[7]).all() and np.isfinite(np.delete(got, 7, axis=0)).all()
    for o in (V, W, C, Vb, Wb, mp, mq):
        o.delete()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m,k,ld", [(5, 5, 5), (8, 8, 8), (13, 7, 17), (16, 16, 16), (24, 20, 24), (31, 31, 33), (32, 32, 32)])
@pytest.mark.parametrize("n", [1, 130, 5003])
def test_product_with_gram(session, n, m, k, ld, dtype):
    """W = a V C + b W with W'W, and W = W C in place with W'W"""
    from phist_b200 import kernels as K
    from phist_b200.objects import SdMat, fn
    rng = np.random.default_rng(n + m)
    eps = np.finfo(dtype).eps
    mp, Vb, V, v = _block(n, ld, 0, m, rng, dtype)
    mq, Wb, W, w = _block(n, k, 0, k, rng, dtype)
    c = (rng.uniform(-1, 1, (m, k)) / m).astype(dtype)
    C, G = SdMat(m, k, dtype).set(c), SdMat(k, k, dtype)
    K.chk(fn(dtype, "fused_mvsd_mvTmv"), 0.5, V.h, C.h, -0.5, W.h, G.h)
    new = W.get().astype(np.float64)
    assert np.abs(new - (0.5 * (v @ c.astype(np.float64)) - 0.5 * w)).max() <= (m + 3) * 2 * eps
    g = G.get()
    assert np.abs(g - new.T @ new).max() <= (n + 3) * (n * np.finfo(np.float64).eps + eps)
    assert np.array_equal(g, g.T) and np.array_equal(G.host(), g)
    X = Vb.view(0, k - 1)
    D = SdMat(k, k, dtype).set(np.eye(k))
    K.chk(fn(dtype, "fused_mvsdi_mvTmv"), 2.0, X.h, V.h, C.h, 1.0, D.h)
    new = X.get().astype(np.float64)
    assert np.abs(new - v @ c.astype(np.float64)).max() <= (m + 3) * 2 * eps
    assert np.abs(D.get() - (2.0 * new.T @ new + np.eye(k))).max() <= 2 * (n + 3) * (n * np.finfo(np.float64).eps + eps)
    for o in (X, D, V, W, C, G, Vb, Wb, mp, mq):
        o.delete()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("mv,k,off", [(1, 4, 0), (8, 4, 0), (9, 4, 0), (20, 4, 0), (10, 2, 1), (37, 3, 1), (64, 1, 0), (16, 16, 0),
                                      (24, 24, 0), (32, 32, 0), (64, 32, 0), (33, 33, 1), (40, 64, 0), (64, 64, 0),
                                      (17, 18, 0), (32, 56, 0), (16, 32, 0)])
@pytest.mark.parametrize("n", [0, 1, 64, 65, 5003])
def test_in_place_product_with_another_block(session, n, mv, k, off, dtype):
    """W = W C in place and D = a V'W + b D of the new W, V another block.  A
    row of W is a sum of k products of size at most 1/k; the sum over n rows of
    products of size at most 1 rounds by at most n eps per term in FP32"""
    from phist_b200 import kernels as K
    from phist_b200.objects import SdMat, fn
    rng = np.random.default_rng(n + mv + k)
    eps = np.finfo(dtype).eps
    mp, Vb, V, v = _block(n, mv + 2 * off, off, mv, rng, dtype)
    mq, Wb, W, w = _block(n, k + 2 * off, off, k, rng, dtype)
    c = (rng.uniform(-1, 1, (k, k)) / k).astype(dtype)
    d0 = rng.uniform(-1, 1, (mv, k)).astype(dtype)
    C, D = SdMat(k, k, dtype).set(c), SdMat(mv, k, dtype).set(d0)
    K.chk(fn(dtype, "fused_mvsdi_mvTmv"), 0.5, V.h, W.h, C.h, 2.0, D.h)
    new = W.get().astype(np.float64)
    assert np.abs(new - w @ c.astype(np.float64)).max(initial=0) <= (k + 3) * 2 * eps
    terms = np.abs(v).T @ np.abs(new)
    assert (np.abs(D.get() - (0.5 * v.T @ new + 2.0 * d0)) <= (n + 3) * eps * (terms + 4)).all()
    for o in (V, W, C, D, Vb, Wb, mp, mq):
        o.delete()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m,k", [(1, 1), (4, 1), (3, 2), (4, 4), (8, 4)])
@pytest.mark.parametrize("n", [(1 << 19) + 3, (1 << 20) + 3])
def test_thin_product_with_gram_of_many_rows(session, n, m, k, dtype):
    """where the fused W'W of thin blocks changes its kernel; bounds as above"""
    from phist_b200 import kernels as K
    from phist_b200.objects import SdMat, fn
    rng = np.random.default_rng(m + k)
    eps = np.finfo(dtype).eps
    mp, Vb, V, v = _block(n, m, 0, m, rng, dtype)
    mq, Wb, W, w = _block(n, k, 0, k, rng, dtype)
    c = (rng.uniform(-1, 1, (m, k)) / m).astype(dtype)
    C, G = SdMat(m, k, dtype).set(c), SdMat(k, k, dtype)
    K.chk(fn(dtype, "fused_mvsd_mvTmv"), 0.5, V.h, C.h, -0.5, W.h, G.h)
    new = W.get().astype(np.float64)
    assert np.abs(new - (0.5 * (v @ c.astype(np.float64)) - 0.5 * w)).max() <= (m + 3) * 2 * eps
    g = G.get()
    assert (np.abs(g - new.T @ new) <= (n * np.finfo(np.float64).eps + eps) * (np.abs(new).T @ np.abs(new))).all()
    assert np.array_equal(G.host(), g)
    # W = W C in place with W'W of the new W, the result scaled and added
    S = SdMat(k, k, dtype).set((rng.uniform(-1, 1, (k, k)) / k).astype(dtype))
    old, d0 = new, rng.uniform(-1, 1, (k, k)).astype(dtype)
    G.set(d0)
    K.chk(fn(dtype, "fused_mvsdi_mvTmv"), 0.5, W.h, W.h, S.h, 2.0, G.h)
    new = W.get().astype(np.float64)
    assert np.abs(new - old @ S.get().astype(np.float64)).max() <= (k + 3) * 2 * eps
    terms = 0.5 * (np.abs(new).T @ np.abs(new)) + 2 * np.abs(d0)
    assert (np.abs(G.get() - (0.5 * new.T @ new + 2.0 * d0)) <= (n * np.finfo(np.float64).eps + 2 * eps) * terms).all()
    assert np.array_equal(G.host(), G.get())
    S.delete()
    # the products alone: a lane of the register kernel adds at most 2^20 / (4 *
    # 148 * 256) < 8 products in the precision of the block and a warp its lanes
    # in 5 steps; from there on FP64, rounded once
    D = SdMat(m, k, dtype)
    for x, y, xm, S in ((V, W, v, D), (W, W, new, G)):
        K.chk(fn(dtype, "mvecT_times_mvec"), 1.0, x.h, y.h, 0.0, S.h)
        terms = np.abs(xm).T @ np.abs(new)
        assert (np.abs(S.get() - xm.T @ new) <= (n * np.finfo(np.float64).eps + 15 * eps) * terms).all()
        assert np.array_equal(S.host(), S.get())
    D.delete()
    for o in (V, W, C, G, Vb, Wb, mp, mq):
        o.delete()


@pytest.mark.parametrize("vld,vo,wld,wo", [(4, 0, 4, 0), (8, 4, 12, 4), (8, 2, 4, 0), (4, 0, 6, 0), (5, 1, 8, 4)])
@pytest.mark.parametrize("n", [1, 255, 5003])
def test_four_columns(session, n, vld, vo, wld, wo):
    """4 x 4 in FP64, rows on 32-byte boundaries (moved whole) and off them:
    every form of the row kernel; columns beside the views stay as they are"""
    from phist_b200 import kernels as K
    from phist_b200.objects import SdMat
    rng = np.random.default_rng(n + vld)
    eps = np.finfo(np.float64).eps
    mp, Vb, V, v = _block(n, vld, vo, 4, rng, np.float64)
    mq, Wb, W, w = _block(n, wld, wo, 4, rng, np.float64)
    c, d = rng.uniform(-1, 1, (4, 4)) / 4, rng.uniform(-1, 1, (4, 4)) / 4
    C, D, G = SdMat(4, 4).set(c), SdMat(4, 4).set(d), SdMat(4, 4)

    def check(ref):
        got = Wb.get()
        assert np.abs(got[:, wo:wo + 4] - ref).max() <= 14 * eps
        assert np.isnan(np.delete(got, np.s_[wo:wo + 4], axis=1)).all()
        return got[:, wo:wo + 4]

    K.chk(K.phist_Dmvec_times_sdMat, 0.5, V.h, C.h, 0.0, W.h)
    w = check(0.5 * v @ c)
    K.chk(K.phist_Dmvec_times_sdMat, 0.5, V.h, C.h, 2.0, W.h)
    w = check(0.5 * v @ c + 2.0 * w)
    K.chk(K.phist_Dmvec_times_sdMat_inplace, W.h, D.h)
    w = check(w @ d)
    K.chk(K.phist_Dmvec_times_sdMat_add_mvec_times_sdMat, V.h, C.h, W.h, D.h)
    w = check(v @ c + w @ d)
    K.chk(K.phist_Dfused_mvsdi_mvTmv, 1.0, V.h, W.h, C.h, 0.0, G.h)
    w = check(w @ c)
    assert np.abs(G.get() - v.T @ w).max() <= (n + 3) * (n + 3) * eps
    for o in (V, W, C, D, G, Vb, Wb, mp, mq):
        o.delete()


def test_no_columns_in_the_result(session):
    """a factor of no columns: nothing to form, whatever the other block"""
    from phist_b200 import kernels as K
    from phist_b200.objects import Map, Mvec, SdMat
    mp = Map(1000)
    for mv in (1, 5, 20, 64):
        V, W = Mvec(mp.h, mv), Mvec(mp.h, 4).set(np.ones((1000, 4)))
        C, D = SdMat(4, 0), SdMat(mv, 0)
        K.chk(K.phist_Dfused_mvsdi_mvTmv, 1.0, V.h, W.h, C.h, 0.0, D.h)
        assert (W.get() == 1.0).all()
        for o in (V, W, C, D):
            o.delete()
    mp.delete()
