"""SASAW row kernels at the edges of their instantiations (channel counts 4, 9, 16 and the widths
between, several passes), columns below, at and above a warp (edges side by side, two columns per
lane), rows without edges, one row with all of them, unsorted rows, skipped gradients; against the CPU
oracle at the parity tolerances."""
import numpy as np
import pytest

from conftest import assert_parity
from helpers import run_checker, run_library, to_dev
from mops_b200 import _lib, workloads
from test_parity_gpu import compare

import mops_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kw", [
    dict(E=1, n=1, nA=1, nW2=1, nO2=1, L=1, N=1), dict(E=333, n=7, nA=4, nW2=4, nO2=4, L=3, N=30),
    dict(E=2001, n=40, nA=5, nW2=9, nO2=9, L=16, N=200), dict(E=2001, n=40, nA=9, nW2=9, nO2=9, L=32, N=500),
    dict(E=1500, n=30, nA=9, nW2=16, nO2=10, L=33, N=300), dict(E=1500, n=30, nA=16, nW2=5, nO2=16, L=64, N=300),
    dict(E=3000, n=900, nA=9, nW2=9, nO2=9, L=66, N=100), dict(E=2500, n=50, nA=3, nW2=10, nO2=2, L=9, N=60),
    dict(E=1300, n=20, nA=16, nW2=16, nO2=16, L=70, N=900),
])
@pytest.mark.parametrize("order", ["sorted", "one row", "unsorted"])
def test_shapes(oracle, kw, dtype, order):
    d = workloads.sasaw(**kw)
    r = np.random.default_rng(3)
    if order == "one row":
        d["indices_output_1"][:] = kw["n"] // 2
        d["indices_W_1"][::2] = 0
    elif order == "unsorted":
        d["indices_output_1"] = r.permutation(d["indices_output_1"])
    what = f"sasaw {kw} {order}"
    if dtype == np.float32 and order == "one row":
        # The oracle adds E N / nO terms per element one by one: with E = 2001, N = 500 its f32 error,
        # eps sqrt(1e5) = 2e-5 of an element, exceeds the tolerance. So here it computes in f64 on
        # the f32 inputs; the library's own chains have E terms: eps sqrt(3000) = 3e-6.
        rounded = {k: v.astype(np.float32).astype(np.float64) if isinstance(v, np.ndarray) and
                   v.dtype == np.float64 else v for k, v in d.items()}
        got = run_library("sasaw", to_dev(d, np.float32))
        want = run_checker(oracle, "sasaw", rounded, np.float64)
        for k in want:
            assert_parity(got[k], want[k].astype(np.float32), f"{what}/{k}")
        return
    compare("sasaw", d, dtype, oracle, what=what)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_skipped_gradients(oracle, dtype):
    d = workloads.sasaw(E=3000, n=50, nA=9, nW2=9, nO2=9, L=40, N=300, dtype=dtype)
    t = to_dev(d, dtype)
    idx = [t[k] for k in ("indices_A", "indices_W_1", "indices_W_2", "indices_output_1", "indices_output_2")]
    full = mops_b200.sparse_accumulation_scatter_add_with_weights_vjp(
        t["grad_output"], t["A"], t["B"], t["C"], t["W"], *idx)
    for which in range(3):
        some = mops_b200.sparse_accumulation_scatter_add_with_weights_vjp(
            t["grad_output"], t["A"], t["B"], t["C"], t["W"], *idx,
            **{f"compute_grad_{n}": i == which for i, n in enumerate("ABW")})
        assert [x is None for x in some] == [i != which for i in range(3)]
        scale = full[which].abs().max()  # (sums of the same terms, the edges of a row in any order)
        assert (some[which] - full[which]).abs().max() <= (1e-12 if dtype == np.float64 else 1e-5) * scale


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("shift", ["", "B", "W", "grad_output"])
def test_whole_warps(oracle, dtype, shift):
    """L = 32, rows enough for two blocks per SM; with one operand an element past a 16-byte boundary."""
    d = workloads.sasaw(E=9000, n=3000, nA=9, nW2=9, nO2=10, L=32, N=80, dtype=dtype)
    t = to_dev(d, dtype)
    if shift:
        flat = t[shift].new_empty(t[shift].numel() + 1)
        t[shift] = flat[1:].view(t[shift].shape).copy_(t[shift])
    got, want = run_library("sasaw", t), run_checker(oracle, "sasaw", d, dtype)
    for k in want:
        assert_parity(got[k], want[k], f"sasaw L=32 shifted {shift}/{k}")


def _by_rows(d, dtype, oracle, what):
    """All results against the oracle in f64 on the same operands (its f32 chains are too long for the f32
    tolerance); the gradients must have come from the row kernels."""
    t = to_dev(d, dtype)
    got = run_library("sasaw", t)
    assert any("sasaw_edge_gradients" in k for k in _lib.last_kernels()), (what, _lib.last_kernels())
    rounded = {k: v.astype(dtype).astype(np.float64) if isinstance(v, np.ndarray) and v.dtype == np.float64 else v
               for k, v in d.items()}
    want = run_checker(oracle, "sasaw", rounded, np.float64)
    for k in want:
        assert_parity(got[k], want[k].astype(dtype), f"{what}/{k}")
    return t, got


# shapes that the gradients take by rows: edges side by side (L <= 16), one column per lane, two (f32), whole
# rows of 16-byte pieces (32 and 64), 4, 9 and 16 A channels, one pass over the output channels and several
GRADIENTS = [(np.float32, (4, 9, 16), L) for L in (3, 8, 16, 32, 64, 66)] + \
            [(np.float32, (9, 9, 9), L) for L in (3, 8, 16, 64, 66)] + \
            [(np.float64, (4, 9, 16), L) for L in (3, 8, 16, 32, 33, 64, 66)] + \
            [(np.float64, (9, 9, 9), L) for L in (8, 16)] + [(np.float64, (16, 16, 9), L) for L in (3, 8)]


@pytest.mark.parametrize("dtype,channels,L", GRADIENTS)
@pytest.mark.parametrize("rows", ["even", "half in one", "cubic"])
def test_gradients_by_rows(oracle, dtype, channels, L, rows):
    """The rows of W with about equal numbers of edges, and with so many in some that they are cut."""
    nA, nW2, nO2 = channels
    d = workloads.sasaw(E=30000, n=2500, nA=nA, nW2=nW2, nO2=nO2, L=L, N=100)
    r = np.random.default_rng(4)
    if rows == "half in one":
        d["indices_W_1"][r.permutation(30000)[:15000]] = 77
    elif rows == "cubic":
        d["indices_W_1"][:] = (r.random(30000) ** 3 * 2500).astype(np.int32)
    what = f"sasaw {channels} L={L} {rows}"
    t, got = _by_rows(d, dtype, oracle, what)
    if L != 8:
        return
    idx = [t[k] for k in ("indices_A", "indices_W_1", "indices_W_2", "indices_output_1", "indices_output_2")]
    for which, name in enumerate(("grad_A", "grad_B", "grad_W")):  # one at a time
        some = mops_b200.sparse_accumulation_scatter_add_with_weights_vjp(
            t["grad_output"], t["A"], t["B"], t["C"], t["W"], *idx,
            **{f"compute_grad_{x}": i == which for i, x in enumerate("ABW")})
        assert [x is None for x in some] == [i != which for i in range(3)]
        tol = 1e-12 if dtype == np.float64 else 1e-5
        assert np.abs(some[which].cpu().numpy() - got[name]).max() <= tol * np.abs(got[name]).max(), what


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kw", [dict(E=20000, n=40, L=32), dict(E=9000, n=2, L=66), dict(E=30000, n=900, L=16),
                                dict(E=700, n=3000, L=8)])
@pytest.mark.parametrize("rows", ["even", "half in one", "all in one"])
def test_unsorted_rows(oracle, dtype, kw, rows):
    """Rows of an unsorted index, few, long, cut or without edges; waiting and not."""
    import torch

    import mops_b200.torch as mt
    d = workloads.sasaw(nA=9, nW2=9, nO2=9, N=100, **kw)
    r = np.random.default_rng(6)
    p = r.permutation(d["indices_output_1"])
    if rows != "even":
        p[: kw["E"] // (1 if rows == "all in one" else 2)] = kw["n"] // 2
        p[0] = kw["n"] - 1
    d["indices_output_1"] = p
    t = to_dev(d, dtype)
    rounded = {k: v.astype(dtype).astype(np.float64) if isinstance(v, np.ndarray) and v.dtype == np.float64 else v
               for k, v in d.items()}
    want = run_checker(oracle, "sasaw", rounded, np.float64)
    got = run_library("sasaw", t)
    for k in want:
        assert_parity(got[k], want[k].astype(dtype), f"sasaw unsorted {kw} {rows}/{k}")
    out = mt.sparse_accumulation_scatter_add_with_weights(
        t["A"], t["B"], t["C"], t["W"], t["indices_A"], t["indices_W_1"], t["indices_W_2"],
        t["indices_output_1"], t["indices_output_2"], t["output_size"])
    torch.cuda.synchronize()
    assert_parity(out.cpu().numpy(), want["output"].astype(dtype), f"sasaw unsorted {kw} {rows} asynchronous")


@pytest.mark.parametrize("channels", [(9, 9, 9), (9, 4, 8), (8, 5, 10), (9, 10, 1), (16, 4, 16), (10, 16, 7), (4, 9, 9)])
@pytest.mark.parametrize("L", [10, 16, 18, 32, 64, 70])
def test_sums_by_mma(oracle, channels, L):
    """The f64 sums on the tensor-core instruction: rows of 0 to 11 edges, so that steps of four are cut everywhere by
    rows' ends, long ones, passes over more channels than one takes, tiles with one output; an infinity stays in its row."""
    nA, nW2, nO2 = channels
    lengths = np.concatenate([np.arange(12), np.arange(12)[::-1], [300, 0, 0, 1, 33], np.full(200, 40)])
    n = len(lengths)
    d = workloads.sasaw(E=int(lengths.sum()), n=n, nA=nA, nW2=nW2, nO2=nO2, L=L, N=150)
    d["indices_output_1"] = np.repeat(np.arange(n), lengths).astype(np.int32)
    t = to_dev(d, np.float64)
    idx = [t[k] for k in ("indices_A", "indices_W_1", "indices_W_2", "indices_output_1", "indices_output_2")]

    def forward():
        return mops_b200.sparse_accumulation_scatter_add_with_weights(
            t["A"], t["B"], t["C"], t["W"], *idx, t["output_size"])

    got = forward()
    if nO2 > 1:  # (one output channel and many columns are estimated to be faster by edge)
        assert any("sasaw_sum_rows_mma" in k for k in _lib.last_kernels()), _lib.last_kernels()
    want = run_checker(oracle, "sasaw", d, np.float64)
    assert_parity(got.cpu().numpy(), want["output"], f"sasaw mma {channels} L={L}")
    row = 16  # (among short rows; its neighbours share steps with it)
    t["B"][int(lengths[:row].sum())] = float("inf")
    inf = forward()
    others = np.arange(n) != row
    assert np.array_equal(inf.cpu().numpy()[others], got.cpu().numpy()[others])


@pytest.mark.parametrize("channels", [(9, 9, 9), (4, 9, 3), (8, 16, 9), (9, 3, 8), (1, 2, 1), (9, 9, 5)])
@pytest.mark.parametrize("L", [8, 10, 32, 64])
def test_gradients_by_mma(oracle, channels, L):
    """The f64 gradients of A and B on the tensor-core instruction: rows of W with 0 to 20 edges, so that steps of eight are cut
    everywhere, rows of a window of 96 edges and longer ones, the last columns of an incomplete eight; an infinite
    gradient stays with the edges that read it."""
    nA, nW2, nO2 = channels
    lengths = np.concatenate([np.arange(21), np.arange(21)[::-1], [95, 96, 97, 0, 0, 1, 193, 500], np.full(300, 60)])
    n = len(lengths)
    d = workloads.sasaw(E=int(lengths.sum()), n=n, nA=nA, nW2=nW2, nO2=nO2, L=L, N=100)
    r = np.random.default_rng(8)
    d["indices_W_1"] = r.permutation(np.repeat(np.arange(n), lengths)).astype(np.int32)
    t = to_dev(d, np.float64)
    got = run_library("sasaw", t)
    if channels == (9, 9, 9):
        assert any("sasaw_edge_gradients_mma" in k for k in _lib.last_kernels()), _lib.last_kernels()
    want = run_checker(oracle, "sasaw", d, np.float64)
    for k in want:
        assert_parity(got[k], want[k], f"sasaw gradients mma {channels} L={L}/{k}")
    row = 200
    t["grad_output"][row] = float("inf")
    inf = run_library("sasaw", t)
    others = d["indices_output_1"] != row
    for k in ("grad_A", "grad_B"):
        assert np.array_equal(inf[k][others], got[k][others]), k


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("L", [16, 32, 64, 100])
@pytest.mark.parametrize("rows", ["even", "long", "gaps", "one"])
def test_few_rows(oracle, dtype, L, rows):
    """Fewer rows than six a warp: a block's edges in equal pieces. Rows within one piece, over several, a block's only row,
    rows without edges at pieces' ends; the same bits in every run."""
    r = np.random.default_rng(9)
    lengths = {"even": np.full(300, 61), "long": np.where(np.arange(150) % 50 == 7, 900, 40),
               "gaps": np.where(r.random(1200) < 0.5, 0, 33), "one": np.r_[np.zeros(40), 9000, np.zeros(3)]}[rows].astype(int)
    n = len(lengths)
    d = workloads.sasaw(E=int(lengths.sum()), n=n, nA=9, nW2=9, nO2=10, L=L, N=100)
    d["indices_output_1"] = np.repeat(np.arange(n), lengths).astype(np.int32)
    d["indices_W_1"] = r.permutation(d["indices_output_1"])
    t = to_dev(d, dtype)
    got = run_library("sasaw", t)
    rounded = {k: v.astype(dtype).astype(np.float64) if isinstance(v, np.ndarray) and v.dtype == np.float64 else v
               for k, v in d.items()}
    want = run_checker(oracle, "sasaw", rounded, np.float64)
    for k in want:
        assert_parity(got[k], want[k].astype(dtype), f"sasaw few rows {rows} L={L}/{k}")
    again = run_library("sasaw", t)
    assert np.array_equal(again["output"], got["output"])


@pytest.mark.parametrize("channels", [(9, 10, 13), (9, 13, 10), (9, 16, 13), (9, 16, 16)])
@pytest.mark.parametrize("E,n", [(2000, 40), (60000, 2500)])
@pytest.mark.parametrize("order", ["sorted", "unsorted"])
def test_widest_shared_memory(oracle, channels, E, n, order):
    """f64, up to four columns: the table and rings of the row kernels take all of the shared memory, or just as much as
    there is without the kernels' own variables, forward (13 and more outputs) and gradients (13 and more channels
    of W). Sizes that are estimated to be faster by rows."""
    nA, nW2, nO2 = channels
    d = workloads.sasaw(E=E, n=n, nA=nA, nW2=nW2, nO2=nO2, L=4, N=100)
    if order == "unsorted":
        d["indices_output_1"] = np.random.default_rng(5).permutation(d["indices_output_1"])
    compare("sasaw", d, np.float64, oracle, what=f"sasaw {channels} E={E} {order}")


def _forward(t):
    out = mops_b200.sparse_accumulation_scatter_add_with_weights(
        t["A"], t["B"], t["C"], t["W"], t["indices_A"], t["indices_W_1"], t["indices_W_2"], t["indices_output_1"],
        t["indices_output_2"], t["output_size"])
    return out, _lib.last_kernels()


# (estimates, by edge and by rows: 0.17 and 0.36, 0.31 and 0.41, 0.125 and 0.158, 0.080 and 0.067, 0.16 and 0.10 ms)
@pytest.mark.parametrize("channels,L,E,n,by_edge", [
    ((16, 9, 9), 32, 80000, 40000, True), ((16, 16, 16), 32, 60000, 20000, True), ((9, 9, 9), 32, 90000, 30000, True),
    ((9, 9, 9), 32, 80000, 2500, False), ((4, 9, 4), 64, 60000, 10000, False)])
def test_short_rows(oracle, channels, L, E, n, by_edge):
    """f64, sorted index: rows so short that the coupling per row costs more than the edges go by edge."""
    nA, nW2, nO2 = channels
    d = workloads.sasaw(E=E, n=n, nA=nA, nW2=nW2, nO2=nO2, L=L, N=100)
    got, kernels = _forward(to_dev(d, np.float64))
    assert any("sasaw_fwd_quad" in k for k in kernels) == by_edge, kernels
    assert any("sasaw_sum_rows_mma" in k for k in kernels) != by_edge, kernels
    want = oracle.sasaw(d["A"], d["B"], d["C"], d["W"], d["indices_A"], d["indices_W_1"], d["indices_W_2"],
                        d["indices_output_1"], d["indices_output_2"], nO2)
    assert_parity(got.cpu().numpy(), want, f"sasaw short rows {channels}")


# (estimates, by edge and by rows: 0.43 and 1.63, 0.19 and 0.30, 0.22 and 0.12, 0.15 and 0.09 ms)
@pytest.mark.parametrize("channels,L,E,n,by_edge", [
    ((16, 16, 16), 64, 60000, 45000, True), ((9, 9, 4), 64, 60000, 50000, True), ((9, 9, 9), 32, 120000, 4000, False),
    ((4, 4, 9), 64, 50000, 5000, False)])
def test_short_rows_unsorted(oracle, channels, L, E, n, by_edge):
    """f64, no order in the index: short rows are not sorted but go by edge."""
    nA, nW2, nO2 = channels
    d = workloads.sasaw(E=E, n=n, nA=nA, nW2=nW2, nO2=nO2, L=L, N=100)
    d["indices_output_1"] = np.random.default_rng(7).permutation(d["indices_output_1"])
    got, kernels = _forward(to_dev(d, np.float64))
    # (for a sorted index first, and then again, or by edge)
    assert (sum("sasaw_sum_rows_mma" in k for k in kernels) == 2) != by_edge, kernels
    want = oracle.sasaw(d["A"], d["B"], d["C"], d["W"], d["indices_A"], d["indices_W_1"], d["indices_W_2"],
                        d["indices_output_1"], d["indices_output_2"], nO2)
    assert_parity(got.cpu().numpy(), want, f"sasaw short rows, unsorted {channels}")


# (estimates, by edge and by rows: 57 and 71, 82 and 114, 63 and 73; 970 and 162, 147 and 136 us)
@pytest.mark.parametrize("channels,L,E,n,by_edge", [
    ((9, 9, 9), 32, 1036, 518, True), ((4, 9, 9), 68, 8220, 137, True), ((9, 8, 9), 10, 17400, 870, True),
    ((9, 9, 9), 38, 13200, 66, False), ((4, 9, 9), 32, 60000, 2500, False)])
def test_gradients_by_estimate(oracle, channels, L, E, n, by_edge):
    """f64, few or short rows: by edge, but not where a warp would have a long row of the output to itself."""
    nA, nW2, nO2 = channels
    d = workloads.sasaw(E=E, n=n, nA=nA, nW2=nW2, nO2=nO2, L=L, N=100)
    compare("sasaw", d, np.float64, oracle, what=f"sasaw gradients {channels} E={E}")
    assert any("sasaw_vjp_" in k for k in _lib.last_kernels()) == by_edge, _lib.last_kernels()


@pytest.mark.parametrize("which", ["output", "grad_B", "grad_output"])
def test_results_off_sixteen_bytes(oracle, which):
    """f64 results or gradients an element past a 16-byte boundary, which the tensor-core row kernels do not take: sizes that
    go by rows on their account go by edge then."""
    import torch
    # (estimates, by rows on tensor cores and with multiply-adds, by edge: 107, 154, 131; 157, 233, 186 us)
    nA, nW2, nO2 = (16, 4, 9) if which == "output" else (9, 9, 4)
    n = 10000 if which == "output" else 1500
    d = workloads.sasaw(E=60000, n=n, nA=nA, nW2=nW2, nO2=nO2, L=64, N=100)
    t = to_dev(d, np.float64)
    idx = ("indices_A", "indices_W_1", "indices_W_2", "indices_output_1", "indices_output_2")
    t.update(output=t["grad_output"].new_empty(n, nO2, 64), grad_A=t["A"].new_empty(t["A"].shape),
             grad_B=t["B"].new_empty(t["B"].shape), grad_W=t["W"].new_empty(t["W"].shape))
    forward = which == "output"
    first = ("output",) if forward else ("grad_A", "grad_B", "grad_W", "grad_output")
    name = "mops_cuda_sparse_accumulation_scatter_add_with_weights_" + ("f64" if forward else "vjp_f64")
    want = run_checker(oracle, "sasaw", d, np.float64)
    for off in (0, 1):
        if off:
            flat = t[which].new_empty(t[which].numel() + 1)
            t[which] = flat[1:].view(t[which].shape).copy_(t[which])
        torch.cuda.synchronize()
        _lib.call(name, [_lib.make_struct(t[k].data_ptr(), t[k].shape) for k in first + ("A", "B", "C", "W") + idx])
        assert any("sasaw_sum_rows" in k for k in _lib.last_kernels()) == (off == 0), _lib.last_kernels()
        for k in first[:3]:
            assert_parity(t[k].cpu().numpy(), want[k], f"sasaw {which} off by {off}/{k}")


# (nA, nW, nO) by what they have compiled in: groups of four m3, a ninth m3, a ninth m1
@pytest.mark.parametrize("channels,instance", [
    ((8, 9, 3), (1, 0, 0)), ((1, 16, 2), (1, 0, 0)), ((9, 9, 4), (1, 0, 1)), ((9, 16, 3), (1, 0, 1)),
    ((4, 9, 8), (2, 0, 0)), ((3, 16, 7), (2, 0, 0)), ((9, 9, 5), (2, 0, 1)), ((9, 12, 8), (2, 0, 1)),
    ((8, 16, 9), (2, 1, 0)), ((9, 9, 9), (2, 1, 1))])
@pytest.mark.parametrize("L", [8, 32, 34])
@pytest.mark.parametrize("rows", ["whole", "cut"])
def test_every_gradient_kernel(oracle, channels, instance, L, rows):
    """Every instantiation of the f64 gradients of A and B on the tensor-core instruction, at sizes that are estimated to be
    faster by it (1.1 times or more). Rows of W without edges and of one to nine between rows longer than a window of 96 edges, which follow one
    another whole; with one of 300, all are cut into chunks of edges."""
    nA, nW2, nO2 = channels
    lengths = np.tile([0, 0, 1, 3, 8, 9, 25, 95, 96, 97, 128, 128, 0, 60, 100], 160)
    n = len(lengths)  # (2400 rows: whole up to 128 edges)
    if rows == "cut":
        lengths[1200] += 300
    d = workloads.sasaw(E=int(lengths.sum()), n=n, nA=nA, nW2=nW2, nO2=nO2, L=L, N=100)
    d["indices_W_1"] = np.random.default_rng(10).permutation(np.repeat(np.arange(n), lengths)).astype(np.int32)
    got = run_library("sasaw", to_dev(d, np.float64))
    ran = "sasaw_edge_gradients_mma<KS=%d,C9=%d,A9=%d,L=%d>" % (*instance, 32 if nA == 9 and L == 32 else 0)
    assert ran in _lib.last_kernels(), _lib.last_kernels()
    want = run_checker(oracle, "sasaw", d, np.float64)
    for k in want:
        assert_parity(got[k], want[k], f"sasaw gradients {channels} L={L} {rows}/{k}")


@pytest.mark.parametrize("channels", [(9, 9, 9), (4, 4, 5), (16, 4, 9), (9, 4, 1)])
@pytest.mark.parametrize("L", [16, 34, 64, 96])
@pytest.mark.parametrize("rows", ["even", "aligned", "long", "gaps", "one"])
def test_sums_in_pieces(oracle, channels, L, rows):
    """The f64 sums on the tensor-core instruction where a block has fewer than 72 rows and slices of sixteen columns: its edges in 12, 4, 3
    or 2 pieces per slice, for which there is room beside the table and the rings. Rows of several pieces, a row as long as a piece or
    two of them, a block's only row, rows without edges; the same bits in every run. nO = 1: a tile of one output."""
    nA, nW2, nO2 = channels
    r = np.random.default_rng(9)
    lengths = {"even": np.full(300, 61), "aligned": np.full(592, 24), "long": np.where(np.arange(150) % 50 == 7, 900, 40),
               "gaps": np.where(r.random(1200) < 0.5, 0, 33), "one": np.r_[np.zeros(40), 9000, np.zeros(3)]}[rows].astype(int)
    n = len(lengths)
    d = workloads.sasaw(E=int(lengths.sum()), n=n, nA=nA, nW2=nW2, nO2=nO2, L=L, N=100)
    d["indices_output_1"] = np.repeat(np.arange(n), lengths).astype(np.int32)
    t = to_dev(d, np.float64)

    def room(kernels):
        return [int(k.split("PIECES=")[1]) for k in kernels if "sasaw_sum_rows_mma" in k]

    got, kernels = _forward(t)
    slices = (L + 15) // 16
    assert room(kernels) and room(kernels)[0] >= 12 // slices * slices, kernels
    want = run_checker(oracle, "sasaw", d, np.float64)
    assert_parity(got.cpu().numpy(), want["output"], f"sasaw pieces {channels} {rows} L={L}")
    for _ in range(3):
        assert np.array_equal(_forward(t)[0].cpu().numpy(), got.cpu().numpy())
    if channels == (9, 9, 9) and rows == "even":  # gW, behind a sort
        d["indices_W_1"] = r.permutation(d["indices_output_1"])
        gradients = run_library("sasaw", to_dev(d, np.float64))
        assert room(_lib.last_kernels())[0] >= 12 // slices * slices, _lib.last_kernels()
        want = run_checker(oracle, "sasaw", d, np.float64)
        for k in want:
            assert_parity(gradients[k], want[k], f"sasaw pieces {channels} {rows} L={L}/{k}")


# (by rows and by edge: 212 and 324, 100 and 146, 164 and 238 us; 755 and 458 us)
@pytest.mark.parametrize("channels,L,E,n,N,by_edge", [
    ((13, 9, 9), 64, 157122, 4155, 33, False), ((14, 9, 9), 66, 21257, 2103, 282, False),
    ((16, 16, 9), 64, 33079, 2610, 461, False), ((16, 9, 9), 52, 158976, 45932, 47, True)])
def test_wide_rows(oracle, channels, L, E, n, N, by_edge):
    """f64, sorted index, ten and more components of A: by rows unless these are short."""
    nA, nW2, nO2 = channels
    d = workloads.sasaw(E=E, n=n, nA=nA, nW2=nW2, nO2=nO2, L=L, N=N)
    got, kernels = _forward(to_dev(d, np.float64))
    assert any("sasaw_fwd_quad" in k for k in kernels) == by_edge, kernels
    assert any("sasaw_sum_rows_mma" in k for k in kernels) != by_edge, kernels
    want = oracle.sasaw(d["A"], d["B"], d["C"], d["W"], d["indices_A"], d["indices_W_1"], d["indices_W_2"],
                        d["indices_output_1"], d["indices_output_2"], nO2)
    assert_parity(got.cpu().numpy(), want, f"sasaw wide rows {channels}")


# (by rows and by edge: 63 and 101, 62 and 93, 63 and 95 us)
@pytest.mark.parametrize("channels,L,E,n,N", [((9, 9, 4), 32, 9595, 50, 470), ((16, 4, 16), 32, 11901, 74, 438),
                                              ((16, 4, 9), 16, 1441, 9, 528)])
def test_few_edges_unsorted(oracle, channels, L, E, n, N):
    """f64, no order in the index, few long rows: sorted, and then by rows."""
    nA, nW2, nO2 = channels
    d = workloads.sasaw(E=E, n=n, nA=nA, nW2=nW2, nO2=nO2, L=L, N=N)
    d["indices_output_1"] = np.random.default_rng(7).permutation(d["indices_output_1"])
    got, kernels = _forward(to_dev(d, np.float64))
    assert "sasaw_sum_rows_mma" in kernels[-1] and (len(kernels) == 2 or "quad" in kernels[0]), kernels
    want = oracle.sasaw(d["A"], d["B"], d["C"], d["W"], d["indices_A"], d["indices_W_1"], d["indices_W_2"],
                        d["indices_output_1"], d["indices_output_2"], nO2)
    assert_parity(got.cpu().numpy(), want, f"sasaw few edges, unsorted {channels}")


# (by rows and by edge: 245 and 367, 130 and 152, 105 and 124 us)
@pytest.mark.parametrize("channels,L,E,n,N", [((9, 13, 9), 16, 35378, 29742, 232), ((9, 16, 4), 32, 65925, 5626, 147),
                                              ((4, 9, 9), 44, 17856, 399, 113)])
def test_gradients_near_the_line(oracle, channels, L, E, n, N):
    """f64 gradients that are a little faster by rows, beside each of the kernels by edge that are not compiled for the widths."""
    nA, nW2, nO2 = channels
    d = workloads.sasaw(E=E, n=n, nA=nA, nW2=nW2, nO2=nO2, L=L, N=N)
    compare("sasaw", d, np.float64, oracle, what=f"sasaw gradients {channels} E={E}")
    assert any("sasaw_edge_gradients_mma" in k for k in _lib.last_kernels()), _lib.last_kernels()
