"""Nine-point grid matrices with any values (honei_b200/csrc/ell_grid9.cu): the products
that leave the column indices unread, bit for bit against the oracle's ELL product
(la/product.hh:148-206), at grids of odd and even size around the rows a thread, a block
and the grid lines take."""
import ctypes

import numpy as np
import pytest
import torch

import honei_b200 as hb
from honei_b200 import DenseVector, SparseMatrixELL, _lib
from honei_b200.inputs import q1_coefficient_operator, uniform

pytestmark = pytest.mark.gpu


def dvec(a):
    return DenseVector(torch.from_numpy(np.ascontiguousarray(a)).cuda())


def same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


def coefficient_case(oracle, cells, npdt):
    op = q1_coefficient_operator(np.power(4.0, uniform(cells * cells, 5, -0.5, 0.5)).reshape(cells, cells), npdt)
    return op, oracle.Ell(op[0], op[1], op[2], op[3], 1, *op[4:])


@pytest.mark.parametrize("cells", [2, 3, 4, 21, 22, 63, 64, 203])
@pytest.mark.parametrize("npdt", [np.float64, np.float32])
def test_modes(oracle, cells, npdt):
    op, ref = coefficient_case(oracle, cells, npdt)
    n = ref.rows
    A = SparseMatrixELL.from_arrays(*op)
    x, b, P = (oracle.uniform(n, s, npdt) for s in (3, 4, 5))
    y = dvec(np.zeros(n, npdt))
    hb.Product.value(y, A, dvec(x))
    want = oracle.ell_spmv(ref, x)
    assert same(y.numpy(), want)
    # an x one element off the allocation's alignment
    xs = torch.zeros(n + 1, dtype=y.elements.dtype, device="cuda")
    xs[1:] = torch.from_numpy(x).cuda()
    hb.Product.value(y, A, DenseVector(xs[1:]))
    assert same(y.numpy(), want)
    d = oracle.ell_defect(ref, b, x)
    norm = torch.zeros(1, dtype=torch.float64, device="cuda")
    hb.Defect.value(y, dvec(b), A, dvec(x), norm2_out=norm)
    assert same(y.numpy(), d)
    exact = float((d.astype(np.float64) ** 2).sum())
    assert abs(float(norm) - exact) <= n * 2.0 ** -52 * exact        # n squares in another order
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.call("hb2_product_dot_ell", A.handle, dvec(x).ptr, y.ptr, ctypes.c_void_p(out.data_ptr()), s)
    assert same(y.numpy(), want)
    terms = want.astype(np.float64) * x.astype(np.float64)
    assert abs(float(out) - terms.sum()) <= n * 2.0 ** -52 * np.abs(terms).sum()
    xx = dvec(x)
    hb.RISmoother.value(A, dvec(P), dvec(b), xx, max_iters=3)
    for _ in range(3):
        x = x + P * oracle.ell_defect(ref, b, x)
    assert same(xx.numpy(), x)


def test_infinite_neighbours_stay_out_of_boundary_rows(oracle):
    """A boundary row reads its own x only, whatever stands next to it."""
    op, ref = coefficient_case(oracle, 20, np.float64)
    m = 21
    x = uniform(m * m, 3)
    x[m + 1], x[5 * m + 1], x[19 * m + 19] = np.inf, np.nan, -np.inf
    y = dvec(np.zeros(m * m))
    hb.Product.value(y, SparseMatrixELL.from_arrays(*op), dvec(x))
    got = y.numpy().reshape(m, m)
    for edge in (np.s_[0, :], np.s_[-1, :], np.s_[:, 0], np.s_[:, -1]):
        assert np.array_equal(got[edge], x.reshape(m, m)[edge])
    want = oracle.ell_spmv(ref, x)
    assert np.array_equal(np.isnan(got.ravel()), np.isnan(want))


def test_other_structures_read_their_columns(oracle):
    """One column moved: not a grid matrix, still the right product."""
    op, _ = coefficient_case(oracle, 30, np.float64)
    n, _, stride, K, Aj, Ax, Arl = op
    Aj = Aj.copy()
    Aj[8 * stride + 40] = n - 1
    ref = oracle.Ell(n, n, stride, K, 1, Aj, Ax, Arl)
    x = uniform(n, 3)
    y = dvec(np.zeros(n))
    hb.Product.value(y, SparseMatrixELL.from_arrays(n, n, stride, K, Aj, Ax, Arl), dvec(x))
    assert same(y.numpy(), oracle.ell_spmv(ref, x))
