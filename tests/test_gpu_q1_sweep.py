"""Q1 sweep passes (honei_b200/csrc/q1_sweep.cuh): several Jacobi sweeps of a Q1 grid
operator in one pass, with the transfers, the defect and the norm around them.  Bit for
bit against the sweeps of math/ri.hh:97-133 formed with the oracle's defect, and inside
the multigrid against the cycle of single passes, which is pinned to the oracle
elsewhere."""
import numpy as np
import pytest
import torch

import honei_b200 as hb
from honei_b200 import DenseVector, SparseMatrixELL
from honei_b200.inputs import q1_coefficient_operator

pytestmark = pytest.mark.gpu


def dvec(a):
    return DenseVector(torch.from_numpy(np.ascontiguousarray(a)).cuda())


def oracle_ell(oracle, op):
    n, cols, stride, K, Aj, Ax, Arl = op
    return oracle.Ell(n, cols, stride, K, 1, Aj, Ax, Arl)


def check_smoother(oracle, A, ref, npdt, sweeps):
    n = ref.rows
    x, b, P = (oracle.uniform(n, s, npdt) for s in (3, 4, 5))
    d = dvec(x)
    hb.RISmoother.value(A, dvec(P), dvec(b), d, temps=[dvec(np.zeros(n, npdt))], max_iters=sweeps)
    for _ in range(sweeps):
        x = x + P * oracle.ell_defect(ref, b, x)       # every product and sum rounded, as the kernels do
    assert np.array_equal(d.numpy().view(np.uint8), x.view(np.uint8))


# strips own 52 (FP64, 20 below m = 400) or 52 to 58 columns, chunks 2 rows and up: grids
# below, at and above one strip and one chunk, up to several blocks
@pytest.mark.parametrize("cells", [2, 3, 19, 20, 51, 52, 53, 64, 117, 403])
@pytest.mark.parametrize("npdt", [np.float64, np.float32])
@pytest.mark.parametrize("sweeps", [2, 4, 9])
def test_smoother_matches_single_sweeps(oracle, cells, npdt, sweeps):
    op = q1_coefficient_operator(np.ones((cells, cells)), npdt)
    ref = oracle_ell(oracle, op)
    check_smoother(oracle, SparseMatrixELL.from_arrays(*op), ref, npdt, sweeps)


# passes of one sweep beside passes of several: as sweep passes up to 181 points a line (the plain
# layout) and, in FP32, from 1,000; as single sweeps between
@pytest.mark.parametrize("cells", [180, 181, 998, 999])
@pytest.mark.parametrize("npdt", [np.float64, np.float32])
@pytest.mark.parametrize("sweeps", [2, 3])
def test_smoother_with_passes_of_one_sweep(oracle, cells, npdt, sweeps):
    op = q1_coefficient_operator(np.ones((cells, cells)), npdt)
    check_smoother(oracle, SparseMatrixELL.from_arrays(*op), oracle_ell(oracle, op), npdt, sweeps)


# either side of the sizes from which a product, a defect and a defect with its norm stream
@pytest.mark.parametrize("cells", [598, 599, 638, 639, 766, 767, 948, 949, 1098, 1099])
@pytest.mark.parametrize("npdt", [np.float64, np.float32])
def test_single_passes(oracle, cells, npdt):
    op = q1_coefficient_operator(np.ones((cells, cells)), npdt)
    ref, A = oracle_ell(oracle, op), SparseMatrixELL.from_arrays(*op)
    x, b = oracle.uniform(ref.rows, 3, npdt), oracle.uniform(ref.rows, 4, npdt)
    xd, bd, y = dvec(x), dvec(b), dvec(np.zeros(ref.rows, npdt))
    hb.Product.value(y, A, xd)
    assert np.array_equal(y.numpy().view(np.uint8), oracle.ell_spmv(ref, x).view(np.uint8))
    d = oracle.ell_defect(ref, b, x)
    hb.Defect.value(y, bd, A, xd)
    assert np.array_equal(y.numpy().view(np.uint8), d.view(np.uint8))
    y, norm2 = dvec(np.zeros(ref.rows, npdt)), torch.zeros(1, dtype=torch.float64, device="cuda")
    hb.Defect.value(y, bd, A, xd, norm2_out=norm2)
    assert np.array_equal(y.numpy().view(np.uint8), d.view(np.uint8))
    # a sum of n squares in FP64 in another order
    exact = float(np.dot(d.astype(np.float64), d.astype(np.float64)))
    assert abs(float(norm2) / exact - 1.0) <= ref.rows * 2.0 ** -52


@pytest.mark.parametrize("npdt", [np.float64, np.float32])
def test_smoother_anisotropic_operator(oracle, npdt):
    """Couplings that differ: the form with one product per slot."""
    dt = torch.float64 if npdt == np.float64 else torch.float32
    for level in (5, 9):
        check_smoother(oracle, SparseMatrixELL.poisson_q1(level, dt, aniso=3.0),
                       oracle.q1_ell(level, npdt, aniso=3.0), npdt, 4)


@pytest.mark.parametrize("row", ["interior", "boundary"])
def test_one_different_row_is_not_a_grid_operator(oracle, row):
    """A matrix that differs from the grid operator in one entry keeps its own rows."""
    cells = 40
    n, _, stride, K, Aj, Ax, Arl = q1_coefficient_operator(np.ones((cells, cells)))
    Ax = Ax.copy()
    Ax[3 * stride + 20 * (cells + 1) + 17 if row == "interior" else cells] *= 1.5
    op = (n, n, stride, K, Aj, Ax, Arl)
    check_smoother(oracle, SparseMatrixELL.from_arrays(*op), oracle_ell(oracle, op), np.float64, 4)


# V-cycles: levels up to 33 points a line and the coarse CG in one block (q1_bottom.cu)
@pytest.mark.parametrize("coarse,level", [(3, 4), (3, 5), (3, 7), (3, 8), (3, 9), (1, 2), (1, 7), (2, 6)])
@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
@pytest.mark.parametrize("pre,post,cycle,aniso", [(4, 4, "V", 1.0), (1, 2, "V", 1.0), (3, 1, "W", 1.0), (5, 9, "V", 1.0),
                                                  (2, 4, "V", 2.0)])
def test_cycle_matches_single_passes(monkeypatch, coarse, level, dt, pre, post, cycle, aniso):
    m = (1 << level) + 1
    i = torch.arange(m * m, device="cuda", dtype=torch.float64)
    out = []
    for flag in ("1", "0"):
        monkeypatch.setenv("HB2_Q1_TRANSFER", flag)       # 0: no transfer or sweep kernels
        data = hb.MGData.poisson_q1(coarse, level, dtype=dt, aniso=aniso,
                                    params=hb.mg_params(pre, post, max_iters=3, eps=1e-30, cycle=cycle))
        x = DenseVector(torch.cos(1.7 * i).to(dt))
        hb.MGSolver.value(data, DenseVector(torch.sin(i).to(dt)), x)
        out.append((x.numpy(), data.rnorm_final))
    assert np.array_equal(out[0][0].view(np.uint8), out[1][0].view(np.uint8))
    # the norms: sums of m^2 squares in two orders, each at most m^2 eps off relative to the sum
    assert abs(out[0][1] / out[1][1] - 1.0) <= m * m * 2.0 ** -52


# The coarse CG on a 9 x 9 Q1 grid operator with equal couplings, three rows of one column a lane
# (cg_warp_grid9), against the one that gathers from the ELL matrix; aniso != 1 and a coarsest of
# another size keep the latter on both sides.  caps: no step, one, fewer and more than it takes.
@pytest.mark.parametrize("coarse,aniso", [(3, 1.0), (3, 2.0), (2, 1.0)])
@pytest.mark.parametrize("cap", [0, 1, 7, 100])
@pytest.mark.parametrize("mixed", [False, True])
def test_coarse_cg_on_the_grid(monkeypatch, coarse, aniso, cap, mixed):
    dt = torch.float32 if mixed else torch.float64
    m = 33
    i = torch.arange(m * m, device="cuda", dtype=torch.float64)
    out = []
    for flag in ("1", "0"):
        monkeypatch.setenv("HB2_Q1_TRANSFER", flag)
        data = hb.MGData.poisson_q1(coarse, 5, dtype=dt, aniso=aniso,
                                    params=hb.mg_params(4, 4, max_iters=2, max_iters_coarse=cap, eps=1e-30,
                                                        coarse_exact=False, coarse_fp64=mixed))
        x = DenseVector(torch.zeros(m * m, device="cuda", dtype=dt))
        hb.MGSolver.value(data, DenseVector(torch.sin(i).to(dt)), x)
        out.append(x.numpy().astype(np.float64))
    # a coarse solution differs by at most steps x condition (below 64 on 9 x 9) x 2^-52; two cycles
    # add one such correction each.  Stored in FP32 it may round to the neighbour, and then so may
    # each of the at most 24 sweeps and transfers of a cycle behind it.
    u = 2.0 ** -52 * 100 * 64 + (24 * 2.0 ** -23 if mixed else 0.0)
    assert np.abs(out[0] - out[1]).max() <= 2 * 2 * u * np.abs(out[1]).max()


def test_coarsest_operator_with_more_slots(oracle):
    """A coarsest matrix of ten slots (one of them empty) does not fit the bottom block: the levels
    above run as sweep passes beside a coarse CG of their own.  Reference order, so the same bits."""
    m = 33
    i = torch.arange(m * m, device="cuda", dtype=torch.float64)
    ref = oracle.q1_ell(3)
    Aj, Ax = (np.concatenate([a, np.zeros(ref.stride, a.dtype)]) for a in (ref.Aj, ref.Ax))
    wide = SparseMatrixELL.from_arrays(ref.rows, ref.cols, ref.stride, ref.K + 1, Aj, Ax, ref.Arl)
    transfers = [SparseMatrixELL.transfer(level) for level in (4, 5)]
    out = []
    for coarse in (wide, SparseMatrixELL.poisson_q1(3)):
        data = hb.MGData([coarse] + [SparseMatrixELL.poisson_q1(level) for level in (4, 5)], [t[0] for t in transfers],
                         [t[1] for t in transfers], params=hb.mg_params(4, 4, max_iters=3, eps=1e-30, coarse_exact=True))
        x = DenseVector(torch.cos(1.7 * i))
        hb.MGSolver.value(data, DenseVector(torch.sin(i)), x)
        out.append(x.numpy())
    assert np.array_equal(out[0].view(np.uint8), out[1].view(np.uint8))
