"""The tensor-memory kernels of HPE and SAP at the edges of their tiles (128 rows per slot), of their
dispatch (rows per lane, blocks per tile, widths that still fit) and of their record tables (columns
without records, one column, many), against the CPU oracle at the parity tolerances."""
import numpy as np
import pytest

from conftest import assert_parity
from helpers import run_checker, run_library, to_dev
from mops_b200 import _lib, workloads
from test_parity_gpu import compare

import mops_b200 as M

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


def _sap_kernels(t):
    """The main kernels of a forward call and of one for both gradients."""
    idx = (t["indices_A"], t["indices_B"], t["indices_output"])
    M.sparse_accumulation_of_products(t["A"], t["B"], t["C"], *idx, t["output_size"])
    forward = _lib.last_kernels()
    M.sparse_accumulation_of_products_vjp(t["grad_output"], t["A"], t["B"], t["C"], *idx)
    return forward[0], _lib.last_kernels()[0]


FWD, VJP = "sap_fwd_resident<%s,NF=1,W=4>", "sap_vjp_resident<%s,W=4>"
BY_PAIRS = "sap_fwd_resident<%s,NF=2,W={}>"


@pytest.mark.parametrize("kw,f64,f32", [
    # (result rows of whole 128-byte lines lie 16 bytes further apart in shared memory)
    (dict(I=148 * 256, nA=20, nB=6, nO=64, K=1000), (FWD, VJP[:-2] + "2>"),
     (FWD[:-2] + "2>", VJP[:-2] + "2>")),
    (dict(I=148 * 512 + 1, nA=16, nB=4, nO=32, K=600), (FWD, VJP), (FWD, VJP)),  # f32: four rows per lane
    (dict(I=2 * 148 * 256 + 255, nA=9, nB=14, nO=3, K=400), (FWD, VJP), (FWD, VJP)),  # 126 products, few result columns
    (dict(I=148 * 128 + 1, nA=16, nB=8, nO=9, K=500), ("sap_fwd_tmem", VJP[:-2] + "2>"),  # 128 products
     ("sap_fwd_tmem", "sap_vjp_tmem")),                                                 # f32: not a tile for every SM
    (dict(I=148 * 256, nA=32, nB=16, nO=20, K=900), ("sap_fwd_tmem", VJP[:-2] + "2>"),
     (BY_PAIRS.format(2), VJP[:-2] + "2>")),
    (dict(I=148 * 512, nA=32, nB=16, nO=20, K=900), ("sap_fwd_tmem", VJP[:-2] + "2>"),
     (BY_PAIRS.format(4), VJP[:-2] + "2>")),
    (dict(I=148 * 512 + 9, nA=24, nB=9, nO=7, K=300), ("sap_fwd_tmem", VJP), (BY_PAIRS.format(4), VJP)),  # products hardly used
    (dict(I=40001, nA=1, nB=1, nO=2, K=900), (FWD, VJP), (FWD[:-2] + "2>", VJP[:-2] + "2>")),  # one cell: three idle groups
    # odd rows; the last tile ends inside a 16-byte piece
    (dict(I=40003, nA=7, nB=11, nO=33, K=511), (FWD, VJP), (FWD[:-2] + "2>", VJP[:-2] + "2>")),
    (dict(I=20003, nA=7, nB=11, nO=33, K=511), (FWD[:-2] + "2>", VJP[:-2] + "2>"), ("sap_fwd_tmem", "sap_vjp_tmem")),
    (dict(I=20011, nA=32, nB=16, nO=100, K=2000), ("sap_fwd_tmem", "sap_vjp_tmem"), ("sap_fwd_tmem", "sap_vjp_tmem")),
])
@pytest.mark.parametrize("dtype", DTYPES)
def test_sap_resident(oracle, kw, f64, f32, dtype):
    """Batches that fill the GPU: records and results in shared memory (sap_fwd_resident, sap_vjp_resident), with as
    many rows per lane as fit, and the shapes next to them that are not taken."""
    d = workloads.sap(**kw)
    r = np.random.default_rng(7)
    d["indices_output"] = r.permutation(d["indices_output"])
    name = "f64" if dtype == np.float64 else "f32"
    kernels = _sap_kernels(to_dev(d, dtype))
    for got, want in zip(kernels, f64 if dtype == np.float64 else f32):
        assert got.startswith(want % name if "%" in want else want), (kernels, want)
    compare("sap", d, dtype, oracle, what=f"sap {kw}")


@pytest.mark.parametrize("dtype", DTYPES)
def test_sap_resident_in_a_plan_and_with_bad_indices(oracle, dtype):
    """Tables of a plan serve both kernels of the gradients and the forward again; an index out of range is
    reported from either, and the call after it works."""
    d = workloads.sap(I=148 * 512, nA=9, nB=6, nO=17, K=700)
    t = to_dev(d, dtype)
    with M.Plan() as plan:
        first = run_library("sap", t)
        tables = plan.tables
        again = run_library("sap", t)
        assert plan.tables == tables == 2
    assert all("resident" in k for k in _sap_kernels(t))
    want = run_checker(oracle, "sap", d, dtype)
    for k in want:
        assert_parity(first[k], want[k], k)
        assert np.array_equal(first[k], again[k]), k
    for name, size in (("indices_A", 9), ("indices_B", 6), ("indices_output", 17)):
        bad = dict(t, **{name: t[name].clone()})
        bad[name][123] = size
        idx = (bad["indices_A"], bad["indices_B"], bad["indices_output"])
        with pytest.raises(M.MopsError, match=f"Index array {name} "):
            M.sparse_accumulation_of_products(t["A"], t["B"], t["C"], *idx, 17)
        with pytest.raises(M.MopsError, match=f"Index array {name} "):
            M.sparse_accumulation_of_products_vjp(t["grad_output"], t["A"], t["B"], t["C"], *idx)
    got = run_library("sap", t)
    assert all(np.array_equal(first[k], got[k]) for k in first)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("kw,kernel", [
    (dict(I=37889, nA=8, nB=3, nO=9, K=17000), "sap_vjp_cells"),    # records larger than shared memory
    (dict(I=38001, nA=2, nB=7, nO=60, K=16500), "sap_vjp_cells"),   # B the wider operand, the last tile ragged
    (dict(I=37889, nA=25, nB=25, nO=30, K=900), "sap_vjp_tmem"),    # few triplets per cell
])
def test_sap_gradients_by_streamed_cells(oracle, kw, kernel, dtype):
    d = workloads.sap(**kw)
    d["indices_output"] = np.random.default_rng(7).permutation(d["indices_output"])
    assert _sap_kernels(to_dev(d, dtype))[1].startswith(kernel)
    if dtype == np.float32:  # (sums of thousands of terms: see test_f32_sums_of_thousands_of_records)
        rounded = {k: v.astype(np.float32).astype(np.float64) if isinstance(v, np.ndarray) and v.dtype == np.float64
                   else v for k, v in d.items()}
        got, want = run_library("sap", to_dev(d, dtype)), run_checker(oracle, "sap", rounded, np.float64)
        for k in want:
            assert np.abs(got[k] - want[k]).max() <= 1e-5 * np.abs(want[k]).max(), k
        return
    compare("sap", d, dtype, oracle, what=f"sap {kw}")


@pytest.mark.parametrize("dtype", DTYPES)
def test_sap_results_at_odd_addresses(oracle, dtype):
    """Results that start one scalar into an allocation: no bulk copies out of shared memory."""
    import torch
    d = workloads.sap(I=148 * 256 + 5, nA=6, nB=4, nO=9, K=600)
    t = to_dev(d, dtype)
    want = run_checker(oracle, "sap", d, dtype)
    odd = {k: t[x].new_empty(t[x].numel() + 1)[1:].view(t[x].shape)
           for k, x in (("output", "grad_output"), ("grad_A", "A"), ("grad_B", "B"))}
    suffix = "f64" if dtype == np.float64 else "f32"

    def call(name, *tensors):
        _lib.call(f"mops_cuda_{name}_{suffix}", [_lib.make_struct(x.data_ptr(), x.shape) for x in tensors])
        torch.cuda.synchronize()
        return _lib.last_kernels()[0]

    torch.cuda.synchronize()
    rest = (t["A"], t["B"], t["C"], t["indices_A"], t["indices_B"], t["indices_output"])
    assert call("sparse_accumulation_of_products", odd["output"], *rest).startswith("sap_fwd_tmem")
    assert call("sparse_accumulation_of_products_vjp", odd["grad_A"], odd["grad_B"], t["grad_output"],
                *rest).startswith("sap_vjp_cells")
    for k in want:
        assert_parity(odd[k].cpu().numpy(), want[k], k)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("kw,narrow", [
    (dict(nA=4, nB=4, nO=8, K=100), (True, True, True)), (dict(nA=4, nB=4, nO=8, K=600), (False, False, False)),
    (dict(nA=1, nB=7, nO=9, K=60), (True, True, True)), (dict(nA=23, nB=10, nO=8, K=250), (False, False, False)),
    (dict(nA=13, nB=2, nO=3, K=140), (True, True, True)), (dict(nA=20, nB=6, nO=50, K=900), (False, False, False)),
])
def test_narrow_sap(oracle, kw, narrow, dtype):
    """Batches that fill the GPU: narrow operands with few triplets (forward, both gradients, one) stay with the
    kernels that gather from shared memory."""
    d = workloads.sap(I=148 * 128 + 1, **kw)
    d["indices_output"] = np.random.default_rng(7).permutation(d["indices_output"])
    t = to_dev(d, dtype)
    args = (t["grad_output"], t["A"], t["B"], t["C"], t["indices_A"], t["indices_B"], t["indices_output"])
    kernels = list(_sap_kernels(t))
    want = run_checker(oracle, "sap", d, dtype)
    for k in ("grad_A", "grad_B"):
        got = M.sparse_accumulation_of_products_vjp(*args, compute_grad_A=k == "grad_A", compute_grad_B=k == "grad_B")
        kernels.append(_lib.last_kernels()[0])
        assert_parity(got[0 if k == "grad_A" else 1].cpu().numpy(), want[k], k)
    assert tuple("small" in k for k in kernels) == narrow + narrow[-1:], kernels
    compare("sap", d, dtype, oracle, what=f"sap {kw}")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("large", [True, False])
@pytest.mark.parametrize("every", [1, 700])
@pytest.mark.parametrize("op,kw,kernel", [
    ("sap", dict(I=300, nA=20, nB=6, nO=50, K=600), "sap_fwd_tmem"),
    ("sap", dict(I=148 * 512 + 77, nA=20, nB=6, nO=50, K=600), "sap_fwd_resident<f%d,NF=1,W=4>"),
    ("sap", dict(I=148 * 512 + 3, nA=7, nB=1, nO=11, K=700), "sap_fwd_resident<f%d,NF=1,W=4>"),  # more operands than products
    ("sap", dict(I=148 * 256, nA=3, nB=5, nO=60, K=900), "sap_fwd_resident<f%d,NF=1"),
    ("sap", dict(I=148 * 512 + 1, nA=32, nB=16, nO=20, K=900), {4: "sap_fwd_resident<f32,NF=2,W=4>", 8: "sap_fwd_tmem"}),
    ("hpe", dict(I=300, N=20, J=300, K=2), "hpe_fwd_tmem"), ("hpe", dict(I=20001, N=20, J=300, K=3), "hpe_fwd_tmem"),
])
def test_products_of_operands_out_of_range(oracle, op, kw, kernel, every, large, dtype):
    """Terms C a b within the range of the type with products a b that are not: A and B times 2^k, C over 2^k, for
    all rows or for few of a tile, which multiplies their sums by exactly 2^k (the other rows' by 2^-k);
    `large` False: -k, where the products underflow. HPE: the forward of order 2, the gradients of order 3."""
    size = np.dtype(dtype).itemsize
    k = (83 if size == 4 else 660) * (1 if large else -1)
    d = workloads.__dict__[op](**kw)
    if op == "hpe":
        d["grad_output"] = np.ones_like(d["grad_output"])
    d = {n: v.astype(dtype) if isinstance(v, np.ndarray) and v.dtype == np.float64 else v for n, v in d.items()}
    d["A"][::5, 0] = 0
    want = run_checker(oracle, op, {n: v.astype(np.float64) if isinstance(v, np.ndarray) and v.dtype == dtype else v
                                    for n, v in d.items()}, np.float64)
    scaled = np.zeros(kw["I"], dtype=bool)
    scaled[kw["I"] // 3 % every::every] = True
    d["C"] = np.ldexp(d["C"], -k)
    for name in ("A", "B") if op == "sap" else ("A",):
        d[name][scaled] = np.ldexp(d[name][scaled], k)
    t = to_dev(d, dtype)
    if op == "sap":
        got = M.sparse_accumulation_of_products(t["A"], t["B"], t["C"], t["indices_A"], t["indices_B"],
                                                t["indices_output"], t["output_size"])
        name = kernel[size] if isinstance(kernel, dict) else kernel % (8 * size) if "%" in kernel else kernel
        want = want["output"]
    elif kw["K"] == 2:
        got, name = M.homogeneous_polynomial_evaluation(t["A"], t["C"], t["indices_A"]), kernel
        want = want["output"]
    else:
        got, name = M.homogeneous_polynomial_evaluation_vjp(t["grad_output"], t["A"], t["C"], t["indices_A"]), "hpe_vjp_tmem"
        want = want["grad_A"]
    assert any(x.startswith(name) for x in _lib.last_kernels()), _lib.last_kernels()
    got = got.cpu().numpy().astype(np.float64)
    got = np.ldexp(got, np.where(scaled, -k, k).reshape((-1,) + (1,) * (got.ndim - 1)))
    assert_parity(got.astype(dtype), want.astype(dtype), f"{op} {kw}")


@pytest.mark.parametrize("kw,kernel", [(dict(I=148 * 256 + 31, nA=20, nB=6, nO=50, K=700), "sap_fwd_resident<f64,NF=1,W=4>"),
                                       (dict(I=148 * 128 + 31, nA=9, nB=11, nO=20, K=500), "sap_fwd_resident<f64,NF=1,W=2>"),
                                       (dict(I=148 * 256 + 31, nA=16, nB=11, nO=30, K=900), "sap_fwd_tmem")])
def test_sap_rows_do_not_depend_on_the_batch(kw, kernel):
    """f64 forward: the same bits for a row in a large batch and in a small one, next to rows whose products of
    operands overflow or underflow, and for these rows themselves."""
    import torch
    d = workloads.sap(**kw)
    d["C"] = np.ldexp(d["C"], -400)
    for row, a, b in ((1010, 600, -600), (1077, 660, 660), (1080, -300, -300), (kw["I"] - 3, 700, 400), (kw["I"] - 9, -400, -660)):
        d["A"][row], d["B"][row] = np.ldexp(d["A"][row], a), np.ldexp(d["B"][row], b)
    t = to_dev(d, np.float64)

    def forward(rows):
        return M.sparse_accumulation_of_products(t["A"][rows].contiguous(), t["B"][rows].contiguous(), t["C"],
                                                 t["indices_A"], t["indices_B"], t["indices_output"], t["output_size"])

    whole = forward(slice(None))
    assert torch.isfinite(whole).all()
    assert _lib.last_kernels()[0].startswith(kernel)
    for rows in (slice(0, 300), slice(1000, 1100), slice(1077, 1078), slice(5000, 9097), slice(kw["I"] - 40, None)):
        part = forward(rows)
        assert _lib.last_kernels()[0].startswith("sap_fwd_tmem")
        assert torch.equal(whole[rows], part), rows


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
