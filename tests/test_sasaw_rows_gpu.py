"""SASAW row kernels at the edges of their instantiations (channel counts 4, 9, 16 and the widths
between, several passes), columns below, at and above a warp (edges side by side, two columns per
lane), rows without edges, one row with all of them, unsorted rows, skipped gradients; against the CPU
oracle at the parity tolerances."""
import numpy as np
import pytest

from conftest import assert_parity
from helpers import run_checker, run_library, to_dev
from mops_b200 import workloads
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
