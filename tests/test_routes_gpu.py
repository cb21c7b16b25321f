"""Which kernels a call launches: the call is captured into a graph, which is
printed, so that nothing runs.  (The results are checked where the operations
are; here it is the choice between equal results.)"""
from __future__ import annotations

import ctypes
import re

import pytest
import torch

import midint

pytestmark = pytest.mark.gpu


@pytest.fixture
def route(ctx, tmp_path):
    """route(call): the names of the kernels that call(stream) launches."""
    cudart = ctypes.CDLL("libcudart.so.13")  # the one that the library is linked with
    stream = torch.cuda.Stream()

    def check(status):
        assert status == 0, status

    def run(call):
        s, graph = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p()
        path = tmp_path / "graph.dot"
        check(cudart.cudaStreamBeginCapture(s, 2))  # relaxed
        try:
            call(stream.cuda_stream)
        finally:
            check(cudart.cudaStreamEndCapture(s, ctypes.byref(graph)))
        check(cudart.cudaGraphDebugDotPrint(graph, str(path).encode(), 1))  # verbose
        check(cudart.cudaGraphDestroy(graph))
        # mangled: a (lower-case) name stands between its length and a capital
        return set(re.findall(r"\d(k_[a-z0-9_]+)(?=[A-Z])", path.read_text()))

    return run


def buffers(words, count=3, offset=0):
    """Buffers of `words` 32-bit words, `offset` words past a 16-byte boundary."""
    keep = [torch.zeros(words + 4, dtype=torch.int32, device="cuda:0") for _ in range(count)]
    return keep, [k.data_ptr() + 4 * offset for k in keep]


@pytest.mark.parametrize("m,kernel", [(28, "k_add"), (29, "k_add"), (30, "k_add_rows"), (48, "k_add_rows"),
                                      (63, "k_add"), (127, "k_add"), (129, "k_add_rows"), (255, "k_add"),
                                      (333, "k_add_rows"), (511, "k_add"), (1001, "k_add"), (4095, "k_add_rows")])
def test_add6_on_unaligned_rows(ctx, route, m, kernel):
    # lengths that fill their group take consecutive limbs per thread
    keep, (a, b, r) = buffers(2 * m * 100, offset=2)
    assert route(lambda s: ctx.add6(a, b, r, 100, m, stream=s)) == {kernel}
    del keep


@pytest.fixture
def own(lib):
    c = midint.Context(0)
    yield c
    c.close()


NTT = {"k_ntt_mul", "k_ntt_mul_cluster", "k_poly_ntt"}


@pytest.mark.parametrize("knob,call,words,m,n", [
    (midint.TUNE_PLAIN_NTT_MIN, "mul", 4, 400, 20), (midint.TUNE_PLAIN_NTT_MIN, "mul_full", 4, 400, 20),
    (midint.TUNE_LO_NTT_MIN, "mul_lo", 2, 200, 20), (midint.TUNE_POLY_NTT_MIN, "poly", 2, 200, 20)])
def test_crossovers_set_by_the_caller_are_exact(own, route, knob, call, words, m, n):
    # small batches, which take the transforms at these lengths by themselves
    keep, (a, b, r) = buffers(words * m * n)

    def names():
        return route(lambda s: getattr(own, call)(a, b, r, n, m, stream=s))

    table = own.get_tuning(knob)
    assert names() <= NTT
    for value in (1025, m + 1):
        own.set_tuning(knob, 0, value)
        assert not names() & NTT, value
    own.set_tuning(knob, 0, m)
    assert names() <= NTT
    own.set_tuning(knob, 0, table)
    assert names() <= NTT
    del keep


CLASSIC = {"k_mul", "k_mul_flex", "k_mul_kara", "k_mul_lo"}
CLUSTER, BLOCKS = {"k_ntt_mul_cluster"}, {"k_ntt_mul"}


@pytest.mark.parametrize("call,m,n,kernels", [
    ("mul", 41, 20, CLASSIC), ("mul", 42, 300, CLUSTER), ("mul", 42, 800, CLASSIC), ("mul", 64, 300, CLUSTER),
    ("mul", 64, 800, CLASSIC), ("mul", 80, 1000, BLOCKS), ("mul", 112, 3000, BLOCKS), ("mul", 124, 1216, BLOCKS),
    ("mul", 128, 60000, CLASSIC), ("mul_full", 42, 800, CLASSIC), ("mul_full", 128, 16384, CLASSIC),
    ("mul_full", 129, 16384, BLOCKS), ("mul_lo", 48, 300, CLUSTER), ("mul_lo", 48, 700, CLASSIC),
    ("mul_lo", 80, 700, CLUSTER), ("mul_lo", 80, 800, CLASSIC), ("mul_lo", 287, 3000, CLASSIC),
    ("mul_lo", 288, 3000, BLOCKS)])
def test_products_by_length_and_batch(own, route, call, m, n, kernels):
    # short products take the transforms only in batches that are faster there
    keep, (a, b, r) = buffers((2 if call == "mul_lo" else 4) * m * n)
    names = route(lambda s: getattr(own, call)(a, b, r, n, m, stream=s))
    assert names and names <= kernels
    del keep
