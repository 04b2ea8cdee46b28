"""SpMMV at block widths that are no power of two, on rows that start on no
vector boundary, and on rows of more than 8 entries: the resident and the
batched kernel (pb_spmmv_pf.cuh) run PHIST's row loop term for term, so their
results equal the one-tile kernel's bit for bit, and the oracle's at 1e-13
(FP32: 1e-5)."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


def _irregular(n, longest, seed):
    rng = np.random.default_rng(seed)
    length = rng.integers(0, longest + 1, n)
    length[0] = longest
    rp = np.concatenate([[0], np.cumsum(length)]).astype(np.int64)
    col = np.concatenate([np.sort(rng.choice(n, m, replace=False)) for m in length]).astype(np.int32)
    return rp, col, rng.uniform(-1, 1, len(col))


@pytest.fixture
def restore(session):
    from phist_b200 import kernels as K
    yield
    K.chk(K.phist_b200_set_spmv_prefetch, 1)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nvec,ld,off", [(1, 3, 1), (2, 2, 0), (2, 5, 1), (3, 3, 0), (4, 9, 1), (5, 5, 0), (6, 6, 0), (7, 9, 2),
                                         (8, 10, 2), (9, 9, 0), (10, 10, 0), (12, 13, 1), (15, 15, 0), (16, 18, 1),
                                         (17, 17, 0), (20, 20, 0), (24, 26, 2), (29, 29, 0), (32, 33, 0), (35, 35, 0)])
@pytest.mark.parametrize("matrix", ["stencil", "irregular"])
def test_any_width(session, oracle, restore, matrix, nvec, ld, off, dtype):
    from phist_b200 import generators as G
    from phist_b200 import kernels as K
    from phist_b200.objects import Mvec, SparseMat, fn
    rp, c, v = G.problem("LAPDIAG3D-11-S3") if matrix == "stencil" else _irregular(1003, 21, 5)
    A = SparseMat.from_crs(rp, c, v, dtype=dtype, flags=K.PHIST_SPARSEMAT_PERM_LOCAL)
    n = len(rp) - 1
    v = v.astype(dtype).astype(np.float64)
    rng = np.random.default_rng(nvec)
    x = np.full((n, ld), np.nan, dtype)
    x[:, off:off + nvec] = rng.uniform(-1, 1, (n, nvec))
    y0 = rng.uniform(-1, 1, (n, nvec)).astype(dtype)
    sh = rng.uniform(-1, 1, nvec).astype(dtype)
    Xb = Mvec(A.domain_map, ld, dtype).set(x)
    X, Y = Xb.view(off, off + nvec - 1), Mvec(A.row_map, nvec, dtype)
    xs = np.ascontiguousarray(x[:, off:off + nvec], np.float64)
    for beta, s in ((0.0, None), (-0.5, sh)):
        ref = oracle.spmmv(rp, c, v, xs, alpha=0.75, beta=beta, y=y0.astype(np.float64),
                           shifts=None if s is None else s.astype(np.float64))
        outs = []
        for pf in (0, 1):
            K.chk(K.phist_b200_set_spmv_prefetch, pf)
            Y.set(y0)
            if s is None:
                K.chk(fn(dtype, "sparseMat_times_mvec"), 0.75, A.h, X.h, beta, Y.h)
            else:
                K.chk(fn(dtype, "sparseMat_times_mvec_vadd_mvec"), 0.75, A.h, K.sptr(s, dtype), X.h, beta, Y.h)
            outs.append(Y.get())
        assert relerr(outs[1], ref) < (1e-13 if dtype == np.float64 else 1e-5)
        assert np.array_equal(outs[0], outs[1])
    for o in (X, Y, Xb, A):
        o.delete()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nvec", [1, 2, 3, 5, 6, 8, 11, 14, 19, 32])
def test_column_dots(session, oracle, nvec, dtype):
    """W'W and V'W per column with the product; sums of n terms of size |y|^2
    and |x||y|, each rounded to n eps of the terms' sum"""
    from phist_b200 import generators as G
    from phist_b200 import kernels as K
    from phist_b200.objects import Mvec, SparseMat, fn
    rp, c, v = G.problem("LAPDIAG3D-11-S3")
    A = SparseMat.from_crs(rp, c, v, dtype=dtype, flags=K.PHIST_SPARSEMAT_PERM_LOCAL)
    n = len(rp) - 1
    x = np.random.default_rng(nvec).uniform(-1, 1, (n, nvec)).astype(dtype)
    X, Y = Mvec(A.domain_map, nvec, dtype).set(x), Mvec(A.row_map, nvec, dtype)
    ww, vw = np.zeros(nvec, dtype), np.zeros(nvec, dtype)
    K.chk(fn(dtype, "fused_spmv_mvdot"), 1.0, A.h, X.h, 0.0, Y.h, K.sptr(ww, dtype), K.sptr(vw, dtype))
    y, xd = Y.get().astype(np.float64), x.astype(np.float64)
    assert relerr(y, oracle.spmmv(rp, c, v, xd)) < (1e-13 if dtype == np.float64 else 1e-5)
    eps = n * np.finfo(dtype).eps
    assert (np.abs(ww - (y * y).sum(0)) <= eps * (y * y).sum(0)).all()
    assert (np.abs(vw - (xd * y).sum(0)) <= eps * np.abs(xd * y).sum(0)).all()
    for o in (X, Y, A):
        o.delete()


def test_many_long_rows(session, oracle, restore):
    """more tiles than one wave of blocks"""
    from phist_b200 import kernels as K
    from phist_b200.objects import Mvec, SparseMat
    rp, c, v = _irregular(30011, 12, 9)
    A = SparseMat.from_crs(rp, c, v, flags=K.PHIST_SPARSEMAT_PERM_LOCAL)
    x = np.random.default_rng(1).uniform(-1, 1, (30011, 4))
    X, Y = Mvec(A.domain_map, 4).set(x), Mvec(A.row_map, 4)
    K.chk(K.phist_DsparseMat_times_mvec, 1.0, A.h, X.h, 0.0, Y.h)
    assert relerr(Y.get(), oracle.spmmv(rp, c, v, x)) < 1e-13
    for o in (X, Y, A):
        o.delete()
