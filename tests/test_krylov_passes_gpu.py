"""The passes of the device GMRES and MINRES (pb_krylov.cuh, pb_spmmv_lz.cuh)
where their forms change: more than 24 basis blocks (several launches), more
than 8 systems (groups of columns; up to the 32 of a call), projection blocks of 16, 17, 32 and 33
columns, no projection, 4 and 8 systems with the dots inside the SpMMV and
the widths beside them, row counts that are no multiple of a tile, restarts,
right-hand sides that are not orthogonal to the projection block.

The iterate after a fixed number of steps is unique; 1e-9 is the bound the
other tests of these solvers hold it to against the same oracle."""
import numpy as np
import pytest

from conftest import relerr
from test_gmres_gpu import _dense, _run, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["gmres", "minres"])
@pytest.mark.parametrize("problem,nq,k,steps,bas", [
    ("LAPDIAG3D-9-S1", 5, 4, 27, 40), ("LAPDIAG3D-9-S1", 16, 8, 10, 10), ("LAPDIAG3D-9-S1", 17, 8, 10, 10),
    ("LAPDIAG3D-9-S2", 32, 4, 6, 6), ("LAPDIAG3D-9-S2", 33, 4, 6, 6), ("LAPDIAG3D-9-S3", 4, 9, 9, 9),
    ("LAPDIAG3D-9-S3", 20, 13, 6, 6), ("LAPDIAG3D-9-S3", 0, 17, 5, 5), ("LAPDIAG3D-10-S4", 3, 1, 12, 5),
    ("LAPDIAG3D-9-S3", 4, 24, 6, 6), ("LAPDIAG3D-9-S3", 4, 25, 6, 4), ("LAPDIAG3D-9-S2", 0, 32, 7, 7),
    ("LAPDIAG3D-10-S4", 3, 5, 8, 8), ("HONEYCOMB-11x7-S3-W1", 2, 8, 7, 7)])
def test_cut_off_iterate(session, oracle, problem, nq, k, steps, bas, solver):
    rp, c, v, Q, R, sigma = _setup(problem, nq, k, 7)
    t, iflag = _run(rp, c, v, Q, R, sigma, 1e-30, steps, bas, solver=solver)
    A = _dense(rp, c, v)
    ref, _ = getattr(oracle, "jada_" + solver)(A, Q, R, sigma, np.full(k, 1e-30), steps, bas)
    assert iflag == k
    assert relerr(t, ref) < 1e-9


@pytest.mark.parametrize("solver", ["gmres", "minres"])
@pytest.mark.parametrize("k", [9, 17, 20])
def test_groups_of_systems(session, solver, k):
    """systems go in even groups of at most eight, whose blocks fill the GPU
    side by side: every system as if it had been passed alone, whatever
    resIndex names (1e-9 as above)"""
    from phist_b200 import generators as G
    rp, c, v = G.problem("LAPDIAG3D-51-S1")
    n = len(rp) - 1
    rng = np.random.default_rng(3)
    Q = np.linalg.qr(rng.standard_normal((n, 4)))[0]
    R = rng.standard_normal((n, 22))
    R -= Q @ (Q.T @ R)
    sigma = rng.uniform(0.5, 1.5, k)
    idx = rng.permutation(22)[:k]
    t, iflag = _run(rp, c, v, Q, R, sigma, 1e-30, 6, 4, res_index=idx, solver=solver)
    assert iflag == k
    for s in range(k):
        ref, iflag = _run(rp, c, v, Q, R, sigma[s:s + 1], 1e-30, 6, 4, res_index=idx[s:s + 1], solver=solver)
        assert iflag == 1 and relerr(t[:, s:s + 1], ref) < 1e-9


@pytest.mark.parametrize("solver", ["gmres", "minres"])
def test_most_systems_single_precision(session, oracle, solver):
    rp, c, v, Q, R, sigma = _setup("LAPDIAG3D-9-S5", 5, 32, 8)
    R *= 1024.0 / np.linalg.norm(R, axis=0)
    t, iflag = _run(rp, c, v, Q, R, sigma, 1e-30, 5, 5, dtype=np.float32, solver=solver)
    ref, _ = getattr(oracle, "jada_" + solver)(_dense(rp, c, v), Q, R, sigma, np.full(32, 1e-30), 5, 5)
    assert iflag == 32 and relerr(t, ref) < 1e-5


@pytest.mark.parametrize("k", [4, 8])
def test_minres_single_precision_dots_in_spmmv(session, oracle, k):
    """FP32: five steps, far from convergence; 1e-5 is the bound for FP32
    kernels against the FP64 oracle"""
    rp, c, v, Q, R, sigma = _setup("LAPDIAG3D-9-S5", 10, k, 8)
    R *= 1024.0 / np.linalg.norm(R, axis=0)
    t, _ = _run(rp, c, v, Q, R, sigma, 1e-30, 5, 5, dtype=np.float32, solver="minres")
    ref, _ = oracle.jada_minres(_dense(rp, c, v), Q, R, sigma, np.full(k, 1e-30), 5, 5)
    assert relerr(t, ref) < 1e-5


def _unprojected(problem, nq, k, seed, part):
    """right-hand sides with `part` of their norm in the span of Q"""
    rp, c, v, Q, R, sigma = _setup(problem, nq, k, seed)
    rng = np.random.default_rng(seed + 1)
    R = R / np.linalg.norm(R, axis=0)
    S = Q @ rng.standard_normal((nq, k))
    R = np.sqrt(1 - part * part) * R + part * S / np.linalg.norm(S, axis=0)
    return rp, c, v, Q, R, sigma


@pytest.mark.parametrize("part", [1e-9, 0.07, 0.6])
@pytest.mark.parametrize("solver,problem,nq,k,steps,bas", [
    ("gmres", "HONEYCOMB-12-S3-W1", 6, 4, 20, 20), ("gmres", "HONEYCOMB-12-S3-W1", 3, 8, 40, 40),
    ("gmres", "LAPDIAG3D-9-S1", 24, 3, 12, 5), ("gmres", "LAPDIAG3D-9-S2", 33, 4, 10, 10),
    ("gmres", "LAPDIAG3D-9-S3", 5, 13, 27, 30), ("minres", "HONEYCOMB-12-S3-W1", 6, 4, 8, 8),
    ("minres", "LAPDIAG3D-9-S1", 3, 8, 8, 8), ("minres", "LAPDIAG3D-9-S1", 24, 3, 8, 4),
    ("minres", "LAPDIAG3D-9-S2", 33, 4, 8, 8), ("minres", "LAPDIAG3D-9-S3", 5, 13, 8, 8)])
def test_right_hand_sides_not_orthogonal_to_q(session, oracle, solver, problem, nq, k, steps, bas, part):
    """Q'V_j enters the first coefficients: the iterate is the oracle's, which
    projects before it orthogonalises"""
    rp, c, v, Q, R, sigma = _unprojected(problem, nq, k, 11, part)
    t, iflag = _run(rp, c, v, Q, R, sigma, 1e-30, steps, bas, solver=solver)
    ref, _ = getattr(oracle, "jada_" + solver)(_dense(rp, c, v), Q, R, sigma, np.full(k, 1e-30), steps, bas)
    assert iflag == k
    assert relerr(t, ref) < 1e-9


@pytest.mark.parametrize("nq,k", [(6, 4), (24, 8)])
def test_residual_estimate_not_orthogonal_to_q(session, oracle, nq, k):
    """a part of the right-hand side outside the operator's range stays in the
    residual: no system may be reported as converged below it"""
    rp, c, v, Q, R, sigma = _unprojected("HONEYCOMB-12-S3-W1", nq, k, 5, 0.3)
    _, iflag = _run(rp, c, v, Q, R, 0 * sigma, 0.29, 60, 60)
    assert iflag == k
    _, iflag = _run(rp, c, v, Q, R, 0 * sigma, 0.35, 60, 60)
    _, conv = oracle.jada_gmres(_dense(rp, c, v), Q, R, 0 * sigma, np.full(k, 0.35), 60, 60)
    assert iflag == k - conv.sum()


@pytest.mark.parametrize("solver", ["gmres", "minres"])
def test_single_precision_not_orthogonal_to_q(session, oracle, solver):
    """FP32 as above, five steps; 1e-5 is the bound for FP32 kernels"""
    rp, c, v, Q, R, sigma = _unprojected("LAPDIAG3D-9-S5", 10, 4, 8, 0.5)
    t, _ = _run(rp, c, v, Q, 1024 * R, sigma, 1e-30, 5, 5, dtype=np.float32, solver=solver)
    ref, _ = getattr(oracle, "jada_" + solver)(_dense(rp, c, v), Q, 1024 * R, sigma, np.full(4, 1e-30), 5, 5)
    assert relerr(t, ref) < 1e-5


@pytest.mark.parametrize("solver", ["gmres", "minres"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_no_rows(session, solver, dtype):
    """a matrix without rows: every residual is zero, all systems converged"""
    for nq in (0, 3):
        t, iflag = _run(np.zeros(1, np.int64), np.zeros(0, np.int32), np.zeros(0), np.zeros((0, nq)), np.zeros((0, 4)),
                        np.ones(4), 1e-6, 5, 5, dtype=dtype, solver=solver)
        assert iflag == 0 and t.shape == (0, 4)
