"""The tensor-memory kernels of HPE and SAP at the edges of their tiles (128 rows per slot), of their
dispatch (rows per lane, blocks per tile, widths that still fit) and of their record tables (columns
without records, one column, many), against the CPU oracle at the parity tolerances."""
import numpy as np
import pytest

from helpers import run_checker, run_library, to_dev
from mops_b200 import workloads
from test_parity_gpu import compare

pytestmark = pytest.mark.gpu
DTYPES = [np.float64, np.float32]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("kw", [
    dict(I=1, N=1, J=1, K=1), dict(I=127, N=3, J=1, K=2), dict(I=129, N=16, J=513, K=4),
    dict(I=1000, N=101, J=700, K=3),       # odd width: rows end inside a sector
    dict(I=300, N=127, J=300, K=4), dict(I=300, N=128, J=300, K=2), dict(I=257, N=203, J=300, K=5),
    dict(I=148 * 128 + 77, N=7, J=90, K=4), dict(I=40000, N=33, J=200, K=3),
    dict(I=515, N=60, J=150, K=10),
])
def test_hpe(oracle, kw, dtype):
    compare("hpe", workloads.hpe(**kw), dtype, oracle, what=f"hpe {kw}")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("kw", [
    dict(I=1, nA=1, nB=1, nO=1, K=3), dict(I=129, nA=20, nB=6, nO=50, K=900),
    dict(I=1000, nA=5, nB=16, nO=33, K=60),   # most cells and several columns receive nothing
    dict(I=148 * 256 + 31, nA=20, nB=6, nO=50, K=1000), dict(I=148 * 128 + 129, nA=3, nB=9, nO=7, K=300),
    dict(I=20000, nA=32, nB=16, nO=99, K=2000), dict(I=19001, nA=16, nB=17, nO=15, K=700),
])
def test_sap(oracle, kw, dtype):
    d = workloads.sap(**kw)
    r = np.random.default_rng(5)
    d["indices_output"] = r.permutation(d["indices_output"])
    d["grad_grad_A"] = r.standard_normal(d["A"].shape)
    d["grad_grad_B"] = r.standard_normal(d["B"].shape)
    compare("sap", d, dtype, oracle, second_order=True, what=f"sap {kw}")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("kw", [
    dict(I=148 * 256, nA=20, nB=6, nO=64, K=1000),         # result rows of whole 128-byte lines: one copy each
    dict(I=148 * 512 + 1, nA=16, nB=4, nO=32, K=600),      # f32: four rows per lane
    dict(I=2 * 148 * 256 + 255, nA=9, nB=14, nO=3, K=400),  # 126 products, few result columns
    dict(I=148 * 128 + 1, nA=16, nB=8, nO=9, K=500),       # 128 products: by pairs, two or four rows per lane
    dict(I=40001, nA=1, nB=1, nO=2, K=50),                 # one cell: three warp groups have nothing to do
    dict(I=40003, nA=7, nB=11, nO=33, K=511),              # odd rows; the last tile ends inside a 16-byte piece
    dict(I=20011, nA=32, nB=16, nO=100, K=2000),
])
def test_sap_resident(oracle, kw, dtype):
    """Batches that fill the GPU: records and results in shared memory (sap_fwd_resident, sap_vjp_resident)."""
    d = workloads.sap(**kw)
    r = np.random.default_rng(7)
    d["indices_output"] = r.permutation(d["indices_output"])
    compare("sap", d, dtype, oracle, what=f"sap {kw}")


@pytest.mark.parametrize("op,kw", [("hpe", dict(I=300, N=13, J=6400, K=4)), ("hpe", dict(I=20000, N=8, J=2000, K=3)),
                                   ("sap", dict(I=100, nA=32, nB=2, nO=3, K=4100)),
                                   ("sap", dict(I=5000, nA=9, nB=15, nO=2, K=2000))])
def test_f32_sums_of_thousands_of_records(oracle, op, kw):
    """Sums in pieces of 32: an error of about eps (sqrt(32) + sqrt(records / 32)) / 2 of the terms' size
    for records of random sign, 4e-7 of the result's norm at most; one chain had 8e-7."""
    d = workloads.__dict__[op](**kw)
    rounded = {k: v.astype(np.float32).astype(np.float64) if isinstance(v, np.ndarray) and v.dtype == np.float64
               else v for k, v in d.items()}
    got = run_library(op, to_dev(d, np.float32))
    want = run_checker(oracle, op, rounded, np.float64)
    for k in want:
        error = np.linalg.norm(got[k].astype(np.float64) - want[k]) / np.linalg.norm(want[k])
        assert error < 4e-7, f"{op} {kw} {k}: {error:.1e}"
