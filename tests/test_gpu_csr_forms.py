"""The forms of the CSR product (honei_b200/csrc/csr.cu): x gathered from global memory or
staged by row window, long rows alone in a CTA (few of them) or four to a CTA (many).  Bit
for bit against the oracle's ordered fma chain (la/product.hh:208-244)."""
import numpy as np
import pytest
import torch

import honei_b200 as hb
from honei_b200 import DenseVector, SparseMatrixCSR
from honei_b200.inputs import uniform

pytestmark = pytest.mark.gpu


# rows around a slice of 32 and a window of 512; long rows of 129 (one chunk and an entry) to
# 4,500 (items past the first 32), one of them up to 200 (four warps a CTA)
@pytest.mark.parametrize("rows,nlong,longest", [(1, 0, 0), (31, 1, 129), (513, 3, 300), (1500, 5, 4500), (6000, 200, 260),
                                               (40000, 2, 500)])
@pytest.mark.parametrize("npdt", [np.float64, np.float32])
@pytest.mark.parametrize("staged,u", [("0", "8"), ("1", "8"), ("1", "16")])
def test_forms(oracle, monkeypatch, rows, nlong, longest, npdt, staged, u):
    monkeypatch.setenv("HB2_CSR_U", u)
    monkeypatch.setenv("HB2_CSR_STAGED", staged)
    rng = np.random.default_rng(rows + nlong)
    length = rng.integers(0, 40, rows)
    where = rng.permutation(rows)[:nlong]
    length[where] = rng.integers(129, longest + 1, nlong) if nlong else 0
    if nlong:
        length[where[0]] = longest
    ar = np.zeros(rows + 1, np.int64)
    np.cumsum(length, out=ar[1:])
    row = np.repeat(np.arange(rows), length)
    cols = rows + 700
    aj = np.clip(row + rng.integers(-300, 700, row.size), 0, cols - 1)
    if rows == 40000:
        aj[row < 512] = rng.integers(0, cols, int((row < 512).sum()))     # one window too wide to stage
    ax = uniform(row.size, 3, dtype=npdt)
    x, b = uniform(cols, 4, dtype=npdt), uniform(rows, 5, dtype=npdt)
    A = SparseMatrixCSR.from_arrays(rows, cols, ar, aj, ax)
    ref = oracle.csr_blocked(rows, cols, ar, aj, ax)
    y = DenseVector(rows, dtype=torch.float64 if npdt == np.float64 else torch.float32)
    xd = DenseVector(torch.from_numpy(x).cuda())
    hb.Product.value(y, A, xd)
    assert np.array_equal(y.numpy().view(np.uint8), oracle.csr_spmv(ref, x).view(np.uint8))
    hb.Defect.value(y, DenseVector(torch.from_numpy(b).cuda()), A, xd)
    assert np.array_equal(y.numpy().view(np.uint8), oracle.csr_defect(ref, b, x).view(np.uint8))


@pytest.mark.parametrize("npdt", [np.float64, np.float32])
@pytest.mark.parametrize("u", ["8", "16"])
@pytest.mark.parametrize("nlong", [1, 5])
def test_few_long_rows_four_to_a_cta(oracle, monkeypatch, npdt, u, nlong):
    """The form of many long rows on a few of them, chosen where the slices gather over all of x."""
    monkeypatch.setenv("HB2_CSR_U", u)
    monkeypatch.setenv("HB2_CSR_DEEP", "0")
    rows = 1500
    rng = np.random.default_rng(nlong)
    length = rng.integers(0, 40, rows)
    length[rng.permutation(rows)[:nlong]] = rng.integers(129, 1400, nlong)
    ar = np.zeros(rows + 1, np.int64)
    np.cumsum(length, out=ar[1:])
    aj = rng.integers(0, rows, int(ar[-1]))
    ax, x = uniform(aj.size, 3, dtype=npdt), uniform(rows, 4, dtype=npdt)
    A = SparseMatrixCSR.from_arrays(rows, rows, ar, aj, ax)
    y = DenseVector(rows, dtype=torch.float64 if npdt == np.float64 else torch.float32)
    hb.Product.value(y, A, DenseVector(torch.from_numpy(x).cuda()))
    ref = oracle.csr_spmv(oracle.csr_blocked(rows, rows, ar, aj, ax), x)
    assert np.array_equal(y.numpy().view(np.uint8), ref.view(np.uint8))
