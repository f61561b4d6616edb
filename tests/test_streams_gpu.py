"""Calls on streams and threads that come and go: the first call of a stream, many short-lived streams,
threads that end with calls in flight; results against the CPU oracle."""
import numpy as np
import pytest

import mops_b200
from conftest import assert_parity
from helpers import to_dev
from mops_b200 import _lib, workloads

pytestmark = pytest.mark.gpu


def _problem(oracle, J=5000, unsorted=True, seed=0):
    d = workloads.opsa(J=J, K=5, L=8, nO=97)
    if unsorted:
        d["indices_output"] = np.random.default_rng(seed).permutation(d["indices_output"])
    want = oracle.opsa(d["A"], d["B"], d["indices_output"], d["output_size"])
    return to_dev(d, np.float64), want


def _call(t):
    return mops_b200.outer_product_scatter_add(t["A"], t["B"], t["indices_output"], t["output_size"])


def test_first_call_of_a_stream_while_the_default_stream_is_busy(oracle):
    """What the call's kernels report to one another (here: the index is not sorted) must not be
    overwritten by the preparation of the stream's status words."""
    import torch
    t, want = _problem(oracle)
    _call(t)
    torch.cuda.synchronize()
    side = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda._sleep(200_000_000)  # about 0.1 s on the default stream
    got = []
    for s in side:
        with torch.cuda.stream(s):
            got.append(_call(t))
    torch.cuda.synchronize()
    for g in got:
        assert_parity(g.cpu().numpy(), want, "first call of a stream")


def test_threads_that_end_with_calls_in_flight(oracle):
    """Asynchronous calls from threads that end at once: their scratch memory stays until the kernels are
    done with it."""
    import threading

    import torch

    import mops_b200.torch as mt
    t, want = _problem(oracle, J=40000)
    filler = torch.randn(4096, 4096, device="cuda")
    got = []

    def work(stream):
        with torch.cuda.stream(stream):
            for _ in range(3):  # (the second call gets a workspace)
                filler @ filler
                got.append(mt.outer_product_scatter_add(t["A"], t["B"], t["indices_output"], t["output_size"]))

    streams = [torch.cuda.Stream() for _ in range(8)]
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
        thread = threading.Thread(target=work, args=(s,))
        thread.start()
        thread.join()
    torch.cuda.synchronize()
    assert len(got) == 24
    for g in got:
        assert_parity(g.cpu().numpy(), want, "thread that ended")


def test_many_short_lived_streams(oracle):
    """A stream per step: states of streams that have gone serve later ones (no allocation is left behind
    per stream), each stream's status words are its own, and calls in flight keep theirs."""
    import ctypes

    import torch

    import mops_b200.torch as mt
    rt = ctypes.CDLL("libcudart.so.12")
    t, want = _problem(oracle)
    s, want_s = _problem(oracle, unsorted=False)

    def steps(n, wait):
        got = []
        for i in range(n):
            handle = ctypes.c_void_p()
            assert rt.cudaStreamCreateWithFlags(ctypes.byref(handle), 1) == 0
            with torch.cuda.stream(torch.cuda.ExternalStream(handle.value)):
                args = t if i % 3 else s
                got.append((_call if wait else mt.outer_product_scatter_add)(
                    *((args,) if wait else (args["A"], args["B"], args["indices_output"], args["output_size"]))))
            assert rt.cudaStreamDestroy(handle) == 0
        torch.cuda.synchronize()
        for i, g in enumerate(got):
            assert_parity(g.cpu().numpy(), want if i % 3 else want_s, f"stream {i}")

    steps(200, wait=False)
    steps(200, wait=True)
    # through the C ABI into one output: torch itself keeps memory for every stream it has seen
    small = to_dev(workloads.opsa(J=20, K=2, L=2, nO=3), np.float64)
    out = torch.empty(3, 2, 2, dtype=torch.float64, device="cuda")
    structs = [_lib.make_struct(x.data_ptr(), x.shape)
               for x in (out, small["A"], small["B"], small["indices_output"])]
    lib = _lib.library()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for i in range(8000):  # (512 bytes each where they are left behind: 4 MB)
        handle = ctypes.c_void_p()
        assert rt.cudaStreamCreateWithFlags(ctypes.byref(handle), 1) == 0
        lib.mops_b200_set_stream(handle)
        try:
            _lib.call("mops_cuda_outer_product_scatter_add_f64", structs)
        finally:
            lib.mops_b200_set_stream(None)
        assert rt.cudaStreamDestroy(handle) == 0
    assert before - torch.cuda.mem_get_info()[0] < 3 << 20
