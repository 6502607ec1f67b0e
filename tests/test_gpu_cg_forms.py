"""The resident forms of the conjugate-gradient solvers: CGSolver NONE on a Q1 grid
operator as one cluster (csrc/cg_cluster.cu, math/cg.hh:64-135) and CGSolver VAR with a
vector P as one cooperative launch (csrc/krylov.cu, math/cg.hh:142-210), at the sizes
where their splits change.  The dots are summed in another order than the reference's, so
a solve may stop a step earlier or later and is held to its own stopping test."""
import ctypes

import numpy as np
import pytest
import torch

import honei_b200 as hb
from honei_b200 import _lib
from honei_b200 import DenseVector, SparseMatrixELL
from honei_b200.inputs import q1_coefficient_operator, uniform

pytestmark = pytest.mark.gpu


def dvec(a):
    return DenseVector(torch.from_numpy(np.ascontiguousarray(a)).cuda())


# one CTA with 1 and 2 nodes a thread (levels 4, 5), 4 and 16 CTAs with 2 and 9 (6, 7, 8)
@pytest.mark.parametrize("level", [4, 5, 6, 7, 8])
@pytest.mark.parametrize("aniso", [1.0, 2.0])
def test_cluster_cg(oracle, level, aniso):
    ref = oracle.q1_ell(level, aniso=aniso)
    b = oracle.ell_spmv(ref, oracle.uniform(ref.rows, 42))
    x0 = 0.1 * oracle.uniform(ref.rows, 7)
    A = SparseMatrixELL.poisson_q1(level, aniso=aniso)
    for start in (np.zeros(ref.rows), x0):
        x = dvec(start)
        _, used, defect = hb.CGSolver.value(A, None, dvec(b), x, 3000, 1e-8)
        _, ref_used = oracle.cg_q1(level, b, x0=start, max_iters=3000, aniso=aniso)[:2]
        r0 = np.linalg.norm(b - oracle.ell_spmv(ref, start))
        assert abs(used - ref_used) <= 1
        # the recursive residual meets the test; the true one follows it to well within a half
        assert defect < 1e-8 * r0
        assert np.linalg.norm(b - oracle.ell_spmv(ref, x.numpy())) < 1.5e-8 * r0


@pytest.mark.parametrize("level", [4, 7, 8])
@pytest.mark.parametrize("cap", [0, 1, 5])
def test_cluster_cg_caps(oracle, level, cap):
    """After a few steps the iterates agree to rounding: a step's sums of n terms, at most
    n eps off, change the iterate by that much relative to its size."""
    ref = oracle.q1_ell(level)
    b = oracle.ell_spmv(ref, oracle.uniform(ref.rows, 42))
    x = dvec(np.zeros(ref.rows))
    _, used, _ = hb.CGSolver.value(SparseMatrixELL.poisson_q1(level), None, dvec(b), x, cap, 1e-8)
    xo = oracle.cg_q1(level, b, max_iters=cap)[0]
    assert used == cap
    assert np.linalg.norm(x.numpy() - xo) <= 2.0 ** -52 * ref.rows * max(1.0, np.linalg.norm(xo))


def test_cluster_cg_f32():
    """FP32 vectors, FP64 dots: the true residual in FP64 is within FP32 rounding of the stop."""
    level, m = 6, 65
    A = SparseMatrixELL.poisson_q1(level, torch.float32)
    b = dvec(uniform(m * m, 3, dtype=np.float32))
    x = DenseVector(m * m, dtype=torch.float32)
    hb.CGSolver.value(A, None, b, x, 2000, 1e-4)
    r = DenseVector(m * m, dtype=torch.float32)
    hb.Defect.value(r, b, A, x)
    # 1e-4 by the recursion, 1e-4 again for its drift over some 200 steps of 6e-8
    assert hb.Norm.value(r) < 2e-4 * hb.Norm.value(b)


# one warp, one CTA, a cluster, and the whole GPU with its grid barrier, which clears the word
@pytest.mark.parametrize("level", [3, 5, 7, 9])
def test_an_expired_wait_of_another_call_is_not_this_solve_s(level):
    """A 1 left in the stream's error word (here from the host) says nothing about a later solve."""
    word = ctypes.c_void_p()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert _lib.load().hb2_workspace_error(stream, ctypes.byref(word)) == 0

    class Word:
        __cuda_array_interface__ = {"shape": (1,), "typestr": "<i4", "data": (word.value, False), "version": 2}
    flag = torch.as_tensor(Word(), device="cuda")
    A = SparseMatrixELL.poisson_q1(level)
    b = dvec(uniform(A.rows(), 3))
    x, y = dvec(np.zeros(A.rows())), dvec(np.zeros(A.rows()))
    used = hb.CGSolver.value(A, None, b, x, 30, 1e-8)[1]
    flag.fill_(1)
    try:
        assert hb.CGSolver.value(A, None, b, y, 30, 1e-8)[1] == used
    finally:
        flag.zero_()
    assert np.array_equal(x.numpy().view(np.uint8), y.numpy().view(np.uint8))


# rows a thread: 1 (one block of 5), 1, 2 and 3
@pytest.mark.parametrize("cells", [47, 100, 350, 449])
@pytest.mark.parametrize("cap", [1, 40])
def test_cg_var_loop(oracle, cells, cap):
    op = q1_coefficient_operator(np.power(4.0, uniform(cells * cells, 5, -0.5, 0.5)).reshape(cells, cells))
    n = op[0]
    ref = oracle.Ell(n, n, op[2], op[3], 1, *op[4:])
    A = SparseMatrixELL.from_arrays(*op)
    P = oracle.jacobi_vector(ref)
    b = oracle.ell_spmv(ref, uniform(n, 42))
    x, used, _ = hb.KrylovSolver(hb.HB2_CG_VAR, A, dvec(P), cap, 0.0).solve(dvec(b), dvec(np.zeros(n)))
    xo, ref_used = oracle.cg_var(ref, P, b, max_iters=cap, eps=0.0)[:2]
    assert used == ref_used == cap
    # dots of n terms in another order: n eps a step, over `cap` steps
    assert np.linalg.norm(x.numpy() - xo) <= 2.0 ** -52 * n * cap * np.linalg.norm(xo)
    s = hb.CGSmoother.value(A, dvec(P), dvec(b), dvec(np.zeros(n)), cap)
    so = oracle.cg_var(ref, P, b, max_iters=cap, eps=0.0, smoother=True)[0]
    assert np.linalg.norm(s.numpy() - so) <= 2.0 ** -52 * n * cap * np.linalg.norm(so)


def loop_against_oracle(oracle, A, ref, cap):
    n = ref.rows
    P = oracle.jacobi_vector(ref)
    b = oracle.ell_spmv(ref, uniform(n, 42))
    x, used, _ = hb.KrylovSolver(hb.HB2_CG_VAR, A, dvec(P), cap, 0.0).solve(dvec(b), dvec(np.zeros(n)))
    xo, ref_used = oracle.cg_var(ref, P, b, max_iters=cap, eps=0.0)[:2]
    assert used == ref_used == cap
    # as above: n eps a step, over `cap` steps
    assert np.linalg.norm(x.numpy() - xo) <= 2.0 ** -52 * n * cap * np.linalg.norm(xo)


# 5, 8, 9 and 13 rows a thread: either side of the instances' limits, and the largest that fits
@pytest.mark.parametrize("cells", [600, 777, 800, 990])
def test_cg_var_loop_with_many_rows_a_thread(oracle, cells):
    op = q1_coefficient_operator(np.power(4.0, uniform(cells * cells, 5, -0.5, 0.5)).reshape(cells, cells))
    ref = oracle.Ell(op[0], op[0], op[2], op[3], 1, *op[4:])
    loop_against_oracle(oracle, SparseMatrixELL.from_arrays(*op), ref, 12)


# a plain matrix that is no grid: nine slots unrolled, and any number of them (two more, empty);
# 1, 2 and 5 rows a thread
@pytest.mark.parametrize("cells", [50, 300, 600])
@pytest.mark.parametrize("slots", [9, 11])
def test_cg_var_loop_on_a_plain_matrix(oracle, monkeypatch, cells, slots):
    monkeypatch.setenv("HB2_ELL_COMPACT", "0")       # the plain layout, and no look for grid operators
    n, _, stride, K, Aj, Ax, Arl = q1_coefficient_operator(
        np.power(4.0, uniform(cells * cells, 5, -0.5, 0.5)).reshape(cells, cells))
    more = np.zeros((slots - K) * stride)
    op = (n, n, stride, slots, np.concatenate([Aj, more.astype(Aj.dtype)]), np.concatenate([Ax, more]), Arl)
    ref = oracle.Ell(n, n, stride, slots, 1, *op[4:])
    loop_against_oracle(oracle, SparseMatrixELL.from_arrays(*op), ref, 12)


# the constant-coefficient operator, whose matrix is ten numbers: 1, 4 and 14 rows a thread, the
# last one beyond the loop's 13
@pytest.mark.parametrize("level", [6, 9, 10])
def test_cg_var_loop_on_the_constant_operator(oracle, level):
    loop_against_oracle(oracle, SparseMatrixELL.poisson_q1(level), oracle.q1_ell(level), 12)
