"""Scatter operations on unsorted indices: one-block and whole-GPU sorts (the line lies at 512
entries) and the one-launch kernels of small problems (up to 2048 and 4096), widths on both sides of a 32-lane row and an 8-row part, rows without entries, one row that
receives everything, against the CPU oracle at the parity tolerances."""
import numpy as np
import pytest

from helpers import run_checker, run_library, to_dev
from mops_b200 import _lib, workloads
from test_parity_gpu import compare

import mops_b200 as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("E,n,K,L", [(2, 2, 1, 1), (511, 7, 4, 33), (2048, 33, 16, 40), (2049, 70, 13, 32), (513, 900, 5, 31), (4097, 1, 9, 32),
                                     (20011, 157, 16, 32), (70001, 40000, 17, 20)])
def test_outer_products(oracle, E, n, K, L, dtype):
    r = np.random.default_rng(E)
    for op, d in (("opsa", workloads.opsa(J=E, K=K, L=L, nO=n)), ("opsaw", workloads.opsaw(E=E, K=K, L=L, n=n))):
        po = r.permutation(d["indices_output"])
        if E > 1000:
            po[::3] = n // 2
        d["indices_output"] = po.astype(np.int32)
        compare(op, d, dtype, oracle, what=f"{op} unsorted {E} {n} {K}x{L}")
        if E < 4096:
            order = np.argsort(d["indices_output"], kind="stable")
            for k in ("A", "B", "indices_output", "indices_W"):
                if k in d:
                    d[k] = d[k][order]
            compare(op, d, dtype, oracle, what=f"{op} sorted {E} {n} {K}x{L}")


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("K,L", [(1, 1), (7, 25), (3, 5), (13, 31), (15, 17), (5, 3)])
def test_gradient_rows_of_odd_sizes(oracle, K, L, dtype):
    """Sorted index, grad_output rows that are no multiple of 16 bytes: every alignment of a row's
    start, and the end of the array inside a 16-byte piece (an odd number of rows)."""
    compare("opsa", workloads.opsa(J=3001, K=K, L=L, nO=57), dtype, oracle, what=f"opsa odd {K}x{L}")
    compare("opsa", workloads.opsa(J=7, K=K, L=L, nO=1), dtype, oracle, what=f"opsa one row {K}x{L}")


def _in_f64(oracle, op, d):
    """The f32 operands' results in f64."""
    rounded = {k: v.astype(np.float32).astype(np.float64) if isinstance(v, np.ndarray) and v.dtype == np.float64
               else v for k, v in d.items()}
    return run_checker(oracle, op, rounded, np.float64)


@pytest.mark.parametrize("E", [200, 512, 513, 4096, 4097])
@pytest.mark.parametrize("order", ["sorted", "one row"])
def test_weighted_f32_sums_carry_f64(oracle, E, order):
    """The precision of the weighted operation does not depend on the number of entries: f64 products and
    sums on both sides of the one-launch kernels' limits, so what is left is the rounding of the
    results, half of 2^-23 each (1.2e-7 of a norm at most; one f32 chain of 512 terms has 1e-6)."""
    d = workloads.opsaw(E=E, K=13, L=32, n=70)
    if order == "one row":
        d["indices_output"][:] = 33
    d["B"][1::2] = -d["B"][::2][: d["B"][1::2].shape[0]] * (1 + 1e-3)  # sums that nearly cancel
    d["A"][1::2] = d["A"][::2][: d["A"][1::2].shape[0]]
    got, want = run_library("opsaw", to_dev(d, np.float32)), _in_f64(oracle, "opsaw", d)
    for k in ("output", "grad_A", "grad_B"):  # (grad_W is added up over entries in f32)
        error = np.linalg.norm(got[k].astype(np.float64) - want[k]) / np.linalg.norm(want[k])
        assert error < 6e-8, f"{E} {order} {k}: {error:.1e}"


@pytest.mark.parametrize("K,L", [(7, 25), (10, 3), (15, 17), (13, 31)])
def test_f32_gradients_of_odd_rows_keep_their_precision(oracle, K, L):
    """grad_output rows that are no multiple of 16 bytes: no less than f32 products (7e-8 of the norm)."""
    d = workloads.opsa(J=7700, K=K, L=L, nO=57)
    t = to_dev(d, np.float32)
    got, want = run_library("opsa", t), _in_f64(oracle, "opsa", d)
    assert any("opsa_vjp_pipe<f32" in k for k in _lib.last_kernels())
    for k in ("grad_A", "grad_B"):
        error = np.linalg.norm(got[k].astype(np.float64) - want[k]) / np.linalg.norm(want[k])
        assert error < 7e-8, f"{K}x{L} {k}: {error:.1e}"


@pytest.mark.parametrize("op", ["opsa", "opsaw"])
@pytest.mark.parametrize("kw", [dict(E=60001, n=31, K=8, L=17), dict(E=40003, n=1000, K=13, L=32), dict(E=9001, n=3, K=5, L=70),
                                dict(E=500, n=90001, K=13, L=32), dict(E=400, n=5, K=3, L=8)])
@pytest.mark.parametrize("rows", ["even", "half in one", "all in one"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_few_and_uneven_rows(oracle, op, kw, rows, dtype):
    """Rows cut by the segments of the gathering kernel, rows of one segment, empty ones."""
    kw = dict(kw)
    E, n = kw.pop("E"), kw.pop("n")
    d = workloads.opsa(J=E, nO=n, **kw) if op == "opsa" else workloads.opsaw(E=E, n=n, **kw)
    po = np.random.default_rng(2).permutation(d["indices_output"])
    if rows != "even":
        po[: E if rows == "all in one" else E // 2] = n // 2
        po[0] = n - 1  # (still not sorted)
    d["indices_output"] = po.astype(np.int32)
    if dtype == np.float32 and rows != "even":
        # the oracle's own f32 chains over one row are too long for the tolerance: f64 on the same operands
        got, want = run_library(op, to_dev(d, dtype)), _in_f64(oracle, op, d)
        for k in want:
            scale = np.abs(want[k]).max()
            assert np.abs(got[k] - want[k]).max() <= 1e-5 * scale, f"{op} {kw} {rows} {k}"
        return
    compare(op, d, dtype, oracle, what=f"{op} {E} {n} {kw} {rows}")


def _streamed(op, t):
    """Which of the two calls take the streaming kernels over a sorted order: forward, gradients."""
    if op == "opsa":
        M.outer_product_scatter_add(t["A"], t["B"], t["indices_output"], t["output_size"])
    else:
        M.outer_product_scatter_add_with_weights(t["A"], t["B"], t["W"], t["indices_W"], t["indices_output"])
    forward = any("gathered" in k for k in _lib.last_kernels())
    if op == "opsa":
        M.outer_product_scatter_add_vjp(t["grad_output"], t["A"], t["B"], t["indices_output"])
    else:
        M.outer_product_scatter_add_with_weights_vjp(t["grad_output"], t["A"], t["B"], t["W"], t["indices_W"],
                                                     t["indices_output"])
    return forward, any("gathered" in k for k in _lib.last_kernels())


def _long_rows(op, E, n, K, L, dtype):
    """Rows for whose gradients the streaming kernels are the faster ones (least_per_row)."""
    if dtype == np.float32 and op == "opsaw":
        least = 16 if L == 32 and K in (9, 13, 16) else None
    elif dtype == np.float32:
        least = 32 if K * L >= 128 and 2 * K * L >= (8 if K <= 8 else 16) * (16 if L <= 16 else 32) else None
    else:
        least = ((4 if op == "opsaw" else 1) if K * L >= 400 else 8 if K * L >= 256 else
                 32 if K * L >= 128 or L >= 24 else None)
    return least is not None and E >= least * n


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("E,n,K,L", [(9001, 160, 16, 32), (9003, 5000, 13, 32), (12005, 77, 9, 32), (30011, 900, 8, 16),
                                     (21001, 300, 9, 20), (70001, 3000, 5, 12), (16007, 1, 7, 28), (3300000, 9, 1, 1)])
def test_streamed_in_sorted_order(oracle, E, n, K, L, dtype):
    """The streaming kernels over a sorted order: rows cut by the warps' shares and rows between them, a
    third of the entries in one row, the last chunk of a share, rows of 4-, 8- and 16-byte pieces."""
    r = np.random.default_rng(E)
    for op, d in (("opsa", workloads.opsa(J=E, K=K, L=L, nO=n)), ("opsaw", workloads.opsaw(E=E, K=K, L=L, n=n))):
        if E > 1000000 and op == "opsaw":
            continue
        po = r.permutation(d["indices_output"])
        po[::3] = n // 2
        po[0], po[1] = n - 1, 0
        d["indices_output"] = po.astype(np.int32)
        t = to_dev(d, dtype)
        got, want = run_library(op, t), _in_f64(oracle, op, d) if dtype == np.float32 else run_checker(oracle, op, d, dtype)
        if n > 1 and L * np.dtype(dtype).itemsize % 16 == 0:
            assert _streamed(op, t) == (True, _long_rows(op, E, n, K, L, dtype))
        for k in want:  # (sums over thousands of entries: see test_few_and_uneven_rows)
            scale = np.abs(want[k]).max()
            tolerance = (1e-12 if dtype == np.float64 else 1e-5) * scale
            assert np.abs(got[k].astype(np.float64) - want[k]).max() <= tolerance, f"{op} {E} {n} {K}x{L} {k}"


def _with_a_gap(op, E, n, K, L):
    """Entries in the first and the last hundred of n rows, in no order, and none between them."""
    d = workloads.opsa(J=E, K=K, L=L, nO=n) if op == "opsa" else workloads.opsaw(E=E, K=K, L=L, n=n)
    r = np.random.default_rng(E)
    rows = r.integers(0, 200, E)
    d["indices_output"] = np.where(rows < 100, rows, n - 200 + rows).astype(np.int32)
    return d


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("op", ["opsa", "opsaw"])
@pytest.mark.parametrize("E,n,K,L", [(70001, 30001, 5, 12), (70001, 1501, 13, 32), (9002, 231, 16, 32)])
def test_rows_without_entries_in_between(oracle, op, E, n, K, L, dtype):
    d = _with_a_gap(op, E, n, K, L)
    t = to_dev(d, dtype)
    assert _streamed(op, t) == (True, K > 5)
    got = run_library(op, t)
    want = _in_f64(oracle, op, d) if dtype == np.float32 else run_checker(oracle, op, d, dtype)
    for k in want:  # (sums over hundreds of entries: see test_few_and_uneven_rows)
        tolerance = (1e-12 if dtype == np.float64 else 1e-5) * np.abs(want[k]).max()
        assert np.abs(got[k].astype(np.float64) - want[k]).max() <= tolerance, k


@pytest.mark.parametrize("op", ["opsa", "opsaw"])
def test_rows_without_entries_take_no_time_of_their_own(op):
    """300 000 entries with 199 800 empty rows between them, against the same entries in 200 rows: the whole
    GPU clears the rows (7 us); a warp that walks over them one by one needs 40 ms."""
    import torch

    def time(d):
        t = to_dev(d, np.float32)
        calls = []
        for _ in range(6):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            run_library(op, t, to_host=False)
            end.record()
            end.synchronize()
            calls.append(start.elapsed_time(end))
        return min(calls)

    d = _with_a_gap(op, 300000, 200000, 5, 12)
    few = dict(d, indices_output=np.where(d["indices_output"] < 100, d["indices_output"],
                                          d["indices_output"] - 199800).astype(np.int32))
    if op == "opsa":
        few["output_size"] = 200
        few["grad_output"] = np.concatenate([d["grad_output"][:100], d["grad_output"][-100:]])
    assert time(d) < 5 * time(few)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("op", ["opsa", "opsaw"])
@pytest.mark.parametrize("K,L", [(13, 32), (16, 20), (8, 16), (5, 8), (12, 32), (1, 4), (9, 20), (1, 24)])
@pytest.mark.parametrize("per_row", [1, 5, 17, 40, 70])
def test_gradients_by_the_lengths_of_rows(oracle, op, K, L, per_row, dtype):
    """Both sides of the lines between the two gradient kernels. (All rows streamed: 300 000 entries of 1 x 4 in as
    many rows, f32, took 197 us instead of 72.)"""
    E = 6007
    n = E // per_row
    d = workloads.opsa(J=E, K=K, L=L, nO=n) if op == "opsa" else workloads.opsaw(E=E, K=K, L=L, n=n)
    d["indices_output"] = np.random.default_rng(1).permutation(d["indices_output"])
    t = to_dev(d, dtype)
    assert _streamed(op, t)[1] == _long_rows(op, E, n, K, L, dtype)
    compare(op, d, dtype, oracle, what=f"{op} {K}x{L} {per_row}")


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("op", ["opsa", "opsaw"])
def test_streamed_in_sorted_order_with_skipped_gradients_plans_and_bad_indices(oracle, op, dtype):
    E, n, K, L = 12007, 150, 13, 32
    d = workloads.opsa(J=E, K=K, L=L, nO=n) if op == "opsa" else workloads.opsaw(E=E, K=K, L=L, n=n)
    d["indices_output"] = np.random.default_rng(3).permutation(d["indices_output"])
    t = to_dev(d, dtype)
    assert _streamed(op, t) == (True, True)
    want = run_checker(oracle, op, d, np.float64)
    with M.Plan():  # (does not keep the table of an unsorted index)
        for _ in range(2):
            compare(op, d, dtype, oracle, what=f"{op} in a plan")
    forward, vjp = ((M.outer_product_scatter_add, M.outer_product_scatter_add_vjp) if op == "opsa" else
                    (M.outer_product_scatter_add_with_weights, M.outer_product_scatter_add_with_weights_vjp))
    names = ("A", "B") if op == "opsa" else ("A", "B", "W")
    index = ("indices_output",) if op == "opsa" else ("indices_W", "indices_output")

    def call(function, tensors, *before, **keep):
        size = (tensors["output_size"],) if function is forward and op == "opsa" else ()
        return function(*before, *[tensors[k] for k in names], *[tensors[k] for k in index], *size, **keep)

    for skipped in names:
        got = call(vjp, t, t["grad_output"], **{f"compute_grad_{k}": k != skipped for k in names})
        assert any("gathered" in k for k in _lib.last_kernels())
        for k, g in zip(names, got):
            assert (g is None) == (k == skipped)
            if g is not None:
                scale = np.abs(want[f"grad_{k}"]).max()
                tolerance = (1e-12 if dtype == np.float64 else 1e-5) * scale
                assert np.abs(g.cpu().numpy().astype(np.float64) - want[f"grad_{k}"]).max() <= tolerance, (skipped, k)
    for name in index:
        for value in (n, -1):
            bad = dict(t, **{name: t[name].clone()})
            bad[name][4321] = value
            with pytest.raises(M.MopsError, match=f"Index array {name} "):
                call(forward, bad)
            with pytest.raises(M.MopsError, match=f"Index array {name} "):
                call(vjp, bad, t["grad_output"])
    compare(op, d, dtype, oracle, what=f"{op} afterwards")
