"""The streaming kernels of OPSA / OPSAW, and what stands in for them where operands are not aligned, at more
entries than the one-launch kernels take (opsa_small.cuh): the kernel that a call is meant to reach is
asserted, so that a change of the dispatch does not empty these tests. CPU oracle, parity tolerances."""
import numpy as np
import pytest

from conftest import assert_parity
from helpers import run_checker, run_library, to_dev
from mops_b200 import _lib, workloads
from test_parity_gpu import DTYPES

import mops_b200 as M

pytestmark = pytest.mark.gpu


def check(op, d, dtype, oracle, forward=None, gradients=None, t=None, what=""):
    t = to_dev(d, dtype) if t is None else t
    if forward:
        if op == "opsa":
            M.outer_product_scatter_add(t["A"], t["B"], t["indices_output"], t["output_size"])
        else:
            M.outer_product_scatter_add_with_weights(t["A"], t["B"], t["W"], t["indices_W"], t["indices_output"])
        assert any(k.startswith(forward) for k in _lib.last_kernels()), (what, _lib.last_kernels())
    got = run_library(op, t)
    if gradients:  # (the last call)
        assert any(k.startswith(gradients) for k in _lib.last_kernels()), (what, _lib.last_kernels())
    want = run_checker(oracle, op, d, dtype)
    for k in want:
        assert_parity(got[k], want[k], f"{op} {what} {k}")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("J,nO", [(4099, 57), (9001, 301), (4101, 2)])
@pytest.mark.parametrize("K,L", [(1, 1), (7, 25), (3, 5), (13, 31), (15, 17), (5, 3)])
def test_gradient_rows_of_odd_sizes(oracle, J, nO, K, L, dtype):
    """grad_output rows that are no multiple of 16 bytes: every alignment of a row's start, and the end of
    the array inside a 16-byte piece."""
    check("opsa", workloads.opsa(J=J, K=K, L=L, nO=nO), dtype, oracle, "opsa_fwd_pipe", "opsa_vjp_pipe",
          what=f"{K}x{L} {J} {nO}")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("K,L", [(1, 1), (7, 25), (13, 31)])
def test_one_gradient_row_of_odd_size(oracle, K, L, dtype):
    d = workloads.opsa(J=4500, K=K, L=L, nO=1)
    t = to_dev(d, dtype)
    gA, gB = M.outer_product_scatter_add_vjp(t["grad_output"], t["A"], t["B"], t["indices_output"])
    assert any(k.startswith("opsa_vjp_pipe") for k in _lib.last_kernels())
    want = run_checker(oracle, "opsa", d, dtype)
    assert_parity(gA.cpu().numpy(), want["grad_A"], "grad_A")
    assert_parity(gB.cpu().numpy(), want["grad_B"], "grad_B")


@pytest.mark.parametrize("seed", list(range(8)))
def test_random_shapes_and_row_lengths(oracle, seed):
    """Widths within the streaming kernels' range, row lengths from empty to many chunks."""
    r = np.random.default_rng(500 + seed)
    K = int(r.integers(1, 17))
    L = int(r.choice([4, 8, 12, 16, 20, 24, 28, 32])) if seed % 2 else int(r.integers(1, 33))
    nO, J = int(r.integers(1, 300)), int(r.integers(4097, 9000))
    weights = r.random(nO) ** 4
    weights[r.random(nO) < 0.3] = 0.0
    weights[0] += 1e-3
    rows = np.sort(r.choice(nO, size=J, p=weights / weights.sum())).astype(np.int32)
    for dtype in DTYPES:
        d = workloads.opsa(J=J, K=K, L=L, nO=nO, seed=seed)
        d["indices_output"] = rows
        check("opsa", d, dtype, oracle, "opsa_fwd_pipe", "opsa_vjp_pipe", what=f"{K}x{L} {J} {nO}")
        d = workloads.opsaw(E=J, K=K, L=L, n=nO, seed=seed)
        d["indices_output"] = rows
        pipe = "opsa_%s_pipe" if L * np.dtype(dtype).itemsize % 16 == 0 else None
        check("opsaw", d, dtype, oracle, pipe and pipe % "fwd", pipe and pipe % "vjp", what=f"{K}x{L} {J} {nO}")


@pytest.mark.parametrize("op", ["opsa", "opsaw"])
@pytest.mark.parametrize("dtype", DTYPES)
def test_operands_at_odd_addresses(oracle, op, dtype):
    """Operands that start one scalar into an allocation: the kernels without bulk copies."""
    d = workloads.opsa(J=5001, K=13, L=20, nO=57) if op == "opsa" else workloads.opsaw(E=5001, K=13, L=32, n=57)
    t = to_dev(d, dtype)
    for name in ("A", "B", "grad_output"):
        flat = t[name].new_empty(t[name].numel() + 1)
        t[name] = flat[1:].view(t[name].shape).copy_(t[name])
    kernel = "opsa_vjp_mma" if dtype == np.float64 else "opsa_vjp_entries"
    check(op, d, dtype, oracle, "opsa_fwd_rows" if dtype == np.float32 else None, kernel, t=t, what="shifted")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("J,nO", [(1, 100000), (500, 100000), (70000, 200001), (300001, 30000)])
def test_rows_without_entries(oracle, J, nO, dtype):
    """Runs of empty rows in front, between and behind, by one entry per thread and by eight."""
    d = workloads.opsa(J=J, K=2, L=4, nO=nO)
    d["indices_output"][: J // 2] //= 2  # (still ascending, a wide gap in the middle)
    check("opsa", d, dtype, oracle, what=f"empty rows {J} {nO}")
