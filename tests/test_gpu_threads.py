"""Two host threads, each on its own stream, and two live handles that share a kernel: what
one of them needs (a kernel's shared-memory limit) must not be taken away by the other.  Every call is held to the bits that it gives alone."""
import ctypes
import threading

import numpy as np
import pytest
import torch

import honei_b200 as hb
from honei_b200 import _lib
from honei_b200 import DenseVector, SparseMatrixCSR, SparseMatrixELL
from honei_b200.inputs import q1_coefficient_operator, uniform

pytestmark = pytest.mark.gpu


def dvec(a):
    return DenseVector(torch.from_numpy(np.ascontiguousarray(a)).cuda())


def in_threads(*work):
    """Runs the callables at the same time, each on a stream of its own; their results."""
    out, errors = [None] * len(work), []
    start = threading.Barrier(len(work))

    def body(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                out[i] = work[i]()
                torch.cuda.current_stream().synchronize()
        except Exception as e:          # re-raised below, in the test's thread
            errors.append(e)
    torch.cuda.synchronize()
    threads = [threading.Thread(target=body, args=(i,)) for i in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
    return out


@pytest.mark.parametrize("npdt", [np.float64, np.float32])
def test_csr_products_of_different_windows(monkeypatch, npdt):
    """Staged products whose windows of x are some 5 KiB and just below 64 KiB."""
    monkeypatch.setenv("HB2_CSR_U", "8")
    monkeypatch.setenv("HB2_CSR_STAGED", "1")
    rows = 4096
    rng = np.random.default_rng(1)

    def make(spread):
        ar = np.arange(rows + 1, dtype=np.int64) * 8
        row = np.repeat(np.arange(rows), 8)
        aj = np.clip(row + rng.integers(-spread, spread + 1, row.size), 0, rows + 16000)
        return SparseMatrixCSR.from_arrays(rows, rows + 16001, ar, aj, uniform(row.size, 3, dtype=npdt))
    # a window spans 512 + 2 spread columns
    mats = [make(40), make((65536 // np.dtype(npdt).itemsize - 600) // 2)]
    x = dvec(uniform(rows + 16001, 4, dtype=npdt))
    ys = [dvec(np.zeros(rows, npdt)) for _ in mats]

    # straight through the C ABI: the two threads' calls have to meet inside the library
    product = _lib.load().hb2_product_csr

    def products(k, count=20000):
        s = torch.cuda.current_stream().cuda_stream
        args = (mats[k].handle, ctypes.c_void_p(x.ptr.value), ctypes.c_void_p(ys[k].ptr.value), ctypes.c_void_p(s))
        for i in range(count):
            assert product(*args) == 0, (i, _lib.load().hb2_last_error())
    alone = []
    for k in (0, 1):
        products(k, 1)
        alone.append(ys[k].numpy().copy())
    in_threads(lambda: products(0), lambda: products(1))
    for k in (0, 1):
        assert np.array_equal(ys[k].numpy().view(np.uint8), alone[k].view(np.uint8))


def test_cluster_cg_of_different_sizes():
    """Solves on clusters with slabs of different size; a launch refused for want of shared
    memory would fall to another form, with other sums."""
    A = [SparseMatrixELL.poisson_q1(level) for level in (6, 7, 8)]
    b = [dvec(uniform(a.rows(), 3)) for a in A]
    x = [dvec(np.zeros(a.rows())) for a in A]

    def solves(k, count=20):
        out = None
        for _ in range(count):
            hb.fill(x[k], 0.0)
            out = hb.CGSolver.value(A[k], None, b[k], x[k], 60, eps_relative=1e-8)
        return out[1:]
    alone, bits = [], []
    for k in range(3):
        alone.append(solves(k, 1))
        bits.append(x[k].numpy().copy())
    together = in_threads(*[lambda k=k: solves(k) for k in range(3)])
    for k in range(3):
        assert together[k] == alone[k]
        assert np.array_equal(x[k].numpy().view(np.uint8), bits[k].view(np.uint8))


# 5 and 7 rows a thread: one instance of the loop kernel with 80 and 112 KiB of shared memory
@pytest.mark.parametrize("order", [(700, 600), (600, 700)])
def test_two_krylov_solvers_of_one_instance(order):
    def make(cells):
        op = q1_coefficient_operator(np.power(4.0, uniform(cells * cells, 5, -0.5, 0.5)).reshape(cells, cells))
        A = SparseMatrixELL.from_arrays(*op)
        P = hb.RISmoother.jacobi_precon(A, 1.0)
        return hb.KrylovSolver(hb.HB2_CG_VAR, A, P, 10, 0.0), dvec(uniform(op[0], 42)), op[0]
    first = make(order[0])
    alone = first[0].solve(first[1], dvec(np.zeros(first[2])))[0].numpy().copy()
    second = make(order[1])
    for s in (first, second, first):
        x = s[0].solve(s[1], dvec(np.zeros(s[2])))[0].numpy()
        if s is first:
            assert np.array_equal(x.view(np.uint8), alone.view(np.uint8))


def test_matrices_made_on_one_stream():
    """Two threads make a constant-coefficient grid operator and a varying one, again and again,
    on the same stream: each keeps its own rows (one was taken for the other now and then when
    the check of the rows kept its reference row in the stream's workspace)."""
    cells = 6
    n = (cells + 1) ** 2
    ops = [q1_coefficient_operator(np.ones((cells, cells))),
           q1_coefficient_operator(np.power(4.0, uniform(cells * cells, 5, -0.5, 0.5)).reshape(cells, cells))]
    x = dvec(uniform(n, 3))
    b, P = dvec(uniform(n, 4)), dvec(np.full(n, 0.25))
    stream = torch.cuda.current_stream()

    def smooth(A):
        y, t = x.copy(), dvec(np.zeros(n))
        return hb.RISmoother.value(A, P, b, y, temps=[t], max_iters=3).elements
    alone = [smooth(SparseMatrixELL.from_arrays(*op)).cpu() for op in ops]

    def make(k, count=1500):
        return [SparseMatrixELL.from_arrays(*ops[k], stream=stream) for _ in range(count)]
    for k, made in enumerate(in_threads(lambda: make(0), lambda: make(1))):
        for A in made:
            assert torch.equal(smooth(A).cpu(), alone[k])
