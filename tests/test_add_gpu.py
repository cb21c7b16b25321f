"""GPU addition vs the oracle, bit-exact, through the C ABI."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import midint
import oracle as O
from carry_data import carry_stress
from conftest import golden

pytestmark = pytest.mark.gpu


def _stream():
    return torch.cuda.current_stream().cuda_stream


def gpu_add(ctx, devmem, a, b, m, limb_bits=64, offset=0):
    n = a.size // m
    words = a.view(np.uint32).size
    ba, pa = devmem.put(a, offset)
    bb, pb = devmem.put(b, offset)
    br, pr = devmem.empty_words(words, offset)
    dc = torch.full((n + 8,), 7, dtype=torch.uint8, device="cuda:0")
    ctx.add(pa, pb, pr, n, m, carry=dc.data_ptr(), limb_bits=limb_bits, stream=_stream())
    torch.cuda.synchronize()
    r = devmem.get(br, words, offset, a.dtype)
    c = dc.cpu().numpy()
    assert (c[n:] == 7).all(), "carry written past the batch"
    assert (br[offset + words:].cpu().numpy() == -1).all(), "result written past the batch"
    return r, c[:n]


U64_SIZES = [1, 2, 3, 4, 5, 7, 8, 16, 31, 32, 33, 63, 64, 65, 100, 128, 129, 255, 256, 257, 1000, 1024, 2047, 4096]


@pytest.mark.parametrize("m", U64_SIZES)
@pytest.mark.parametrize("n", [1, 7, 300])
def test_add_u64_matches_oracle(ctx, devmem, m, n):
    if m * n > 2_000_000:
        pytest.skip("size")
    a, b = carry_stress(n, m, seed=1000 * m + n)
    r, c = gpu_add(ctx, devmem, a, b, m)
    wr, wc = O.add(a, b, m)
    assert np.array_equal(r, wr)
    assert np.array_equal(c, wc)


@pytest.mark.parametrize("m", [1, 3, 5, 9, 31, 127, 129, 255, 1023, 4097, 8191])
@pytest.mark.parametrize("offset", [0, 1])
def test_add_u32_odd_and_unaligned(ctx, devmem, m, offset):
    n = 37
    a, b = carry_stress(n, m, seed=m, dtype=np.uint32)
    r, c = gpu_add(ctx, devmem, a, b, m, limb_bits=32, offset=offset)
    wr, wc = O.add(a, b, m)
    assert np.array_equal(r, wr) and np.array_equal(c, wc)


@pytest.mark.parametrize("m", [2, 64, 128, 4096])
def test_add_u64_unaligned_rows(ctx, devmem, m):
    # 8-byte aligned but not 16-byte aligned buffers take the scalar path
    a, b = carry_stress(9, m, seed=5 + m)
    r, c = gpu_add(ctx, devmem, a, b, m, offset=2)
    r2, c2 = gpu_add(ctx, devmem, a, b, m, offset=6)
    wr, wc = O.add(a, b, m)
    assert np.array_equal(r, wr) and np.array_equal(c, wc)
    assert np.array_equal(r2, wr)


@pytest.mark.parametrize("m", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096])
def test_add_matches_reference_fixtures(ctx, devmem, m):
    g = golden("ref_sweep.npz")
    r, _ = gpu_add(ctx, devmem, g["a"], g["b"], m, limb_bits=32)
    assert np.array_equal(r, g[f"add_{m}"])
    w = golden("ref_worst.npz")
    r, c = gpu_add(ctx, devmem, w[f"wa_{m}"], w[f"wb_{m}"], m, limb_bits=32)
    assert np.array_equal(r, w[f"wadd_{m}"]) and c.all()


def test_add_config_shape_with_worst_case_rows(ctx, devmem):
    import workloads

    a, b = workloads.add_pairs(n=65536, m=64)
    r, c = gpu_add(ctx, devmem, a, b, 64)
    wr, wc = O.batch_u64("add", a, b, 64, threads=8)
    assert np.array_equal(r, wr) and np.array_equal(c, wc)
    assert c[::8].all() and not r.reshape(-1, 64)[::8].any()


def test_add_in_place(ctx, devmem):
    m, n = 64, 50
    a, b = carry_stress(n, m, seed=99)
    ba, pa = devmem.put(a)
    bb, pb = devmem.put(b)
    ctx.add(pa, pb, pa, n, m, stream=_stream())       # r aliases a exactly
    torch.cuda.synchronize()
    assert np.array_equal(devmem.get(ba, a.view(np.uint32).size), O.add(a, b, m, with_carry=False))


def test_add_empty_batch(ctx, devmem):
    ba, pa = devmem.put(np.zeros(8, np.uint64))
    ctx.add(pa, pa, pa, 0, 8, stream=_stream())


@pytest.mark.parametrize("m", [1, 2, 3, 4, 17, 33, 64, 65, 128, 1000, 2048, 4096])
def test_add6_matches_oracle(ctx, devmem, m):
    n = 41
    a, b = carry_stress(n, m, seed=7 * m)
    ba, pa = devmem.put(a)
    bb, pb = devmem.put(b)
    br, pr = devmem.empty_words(a.view(np.uint32).size)
    ctx.add6(pa, pb, pr, n, m, stream=_stream())
    torch.cuda.synchronize()
    assert np.array_equal(devmem.get(br, a.view(np.uint32).size), O.add6(a, b, m))


def test_compat_gpuAdd(lib):
    g = golden("ref_sweep.npz")
    for m in (16, 128, 4096):
        a, b = g["a"], g["b"]
        r = np.zeros_like(a)
        midint.gpuAdd(midint.U32bits, m, a.size // m, a, b, r)
        assert np.array_equal(r, g[f"add_{m}"])
        a64, b64 = a.view(np.uint64), b.view(np.uint64)
        r64 = np.zeros_like(a64)
        midint.gpuAdd(midint.U64bits, m // 2, a64.size // (m // 2), a64, b64, r64)
        assert np.array_equal(r64.view(np.uint32), g[f"add_{m}"])


def test_host_add_with_carry(ctx):
    a, b = carry_stress(1000, 64, seed=3)
    r = np.zeros_like(a)
    c = np.zeros(1000, np.uint8)
    ctx.host_add(a, b, r, c, 1000, 64)
    wr, wc = O.add(a, b, 64)
    assert np.array_equal(r, wr) and np.array_equal(c, wc)


@pytest.mark.parametrize("tb", [16, 32, 64])
@pytest.mark.parametrize("m", [1, 2, 3, 8, 17, 64, 65, 200, 1024, 2049, 4096])
def test_add_every_thread_width(lib, devmem, tb, m):
    """Every bytes-per-thread choice of the tuning table gives the same sums."""
    c = midint.Context(0)
    try:
        for cls in range(13):
            c.set_tuning(midint.TUNE_ADD_THREAD_BYTES, cls, tb)
        a, b = carry_stress(19, m, seed=5 * m + tb)
        ra, ca = O.add(a, b, m)
        r, cc = gpu_add(c, devmem, a, b, m)
        assert np.array_equal(r, ra) and np.array_equal(cc, ca)
        r6 = devmem.empty_words(a.view(np.uint32).size)
        ba, pa = devmem.put(a)
        bb, pb = devmem.put(b)
        c.add6(pa, pb, r6[1], 19, m, stream=_stream())
        torch.cuda.synchronize()
        assert np.array_equal(devmem.get(r6[0], a.view(np.uint32).size), O.add6(a, b, m))
        if m % 2 == 1:  # odd u32 limb counts take the scalar u32 kernel
            a32, b32 = a.view(np.uint32)[: 19 * m], b.view(np.uint32)[: 19 * m]
            r32, c32 = gpu_add(c, devmem, a32, b32, m, limb_bits=32)
            ref32, cref32 = O.add(a32, b32, m)
            assert np.array_equal(r32, ref32) and np.array_equal(c32, cref32)
    finally:
        c.close()


def test_tuning_rejects_bad_values(ctx):
    with pytest.raises(midint.MidintError):
        ctx.set_tuning(midint.TUNE_ADD_THREAD_BYTES, 13, 16)
    with pytest.raises(midint.MidintError):
        ctx.set_tuning(midint.TUNE_ADD_THREAD_BYTES, 3, 24)
    with pytest.raises(midint.MidintError):
        ctx.set_tuning(midint.TUNE_RAGGED_NTT_MIN, 0, 258)
    with pytest.raises(midint.MidintError):
        ctx.set_tuning(99, 0, 1)
    old = ctx.get_tuning(midint.TUNE_PLAIN_NTT_MIN)
    ctx.set_tuning(midint.TUNE_PLAIN_NTT_MIN, 0, 1025)
    assert ctx.get_tuning(midint.TUNE_PLAIN_NTT_MIN) == 1025
    ctx.set_tuning(midint.TUNE_PLAIN_NTT_MIN, 0, old)


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("m", [1, 3, 5, 9, 23, 25, 31, 33, 63, 65, 127, 129, 257, 1001, 2047, 2049, 4095, 8191])
def test_add_rows_of_odd_lengths(ctx, devmem, m, bits):
    # rows that allow no 16-byte access: every group width and rows-per-thread
    # choice, plain (separate, in place, with carries) and 6a + 10b
    if bits == 64 and m > 4096:
        pytest.skip("the multi-block kernel")
    n = 700 if m < 300 else 37
    a, b = carry_stress(n, m, seed=m + bits, dtype=np.uint64 if bits == 64 else np.uint32)
    want, carry = O.add(a, b, m)
    words = a.view(np.uint32).size
    s = torch.cuda.current_stream().cuda_stream
    for inplace in (False, True):
        (ba, pa), (bb, pb), (br, pr) = devmem.put(a), devmem.put(b), devmem.empty_words(words)
        dc = torch.full((n + 8,), 7, dtype=torch.uint8, device="cuda:0")
        ctx.add(pa, pb, pb if inplace else pr, n, m, carry=dc.data_ptr(), limb_bits=bits, stream=s)
        torch.cuda.synchronize()
        assert np.array_equal(devmem.get(bb if inplace else br, words, 0, a.dtype), want)
        assert np.array_equal(dc.cpu().numpy()[:n], carry) and (dc.cpu().numpy()[n:] == 7).all()
        if bits == 64:
            (ba, pa), (bb, pb) = devmem.put(a), devmem.put(b)
            ctx.add6(pa, pb, pa if inplace else pr, n, m, stream=s)
            torch.cuda.synchronize()
            assert np.array_equal(devmem.get(ba if inplace else br, words), O.add6(a, b, m))


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("m", [6, 7, 10, 13, 16, 24, 27, 30, 41, 48, 80, 96, 97, 131, 160, 161, 191, 193, 319, 320, 321,
                               385, 513, 640, 641, 765, 1025, 1281, 1537])
def test_add_rows_per_thread(ctx, devmem, m, bits):
    # the edges of the rows-per-thread rule (2 to 6 rows), even lengths on rows
    # that are off by one limb
    n = 300 if m < 300 else 29
    a, b = carry_stress(n, m, seed=m + bits, dtype=np.uint64 if bits == 64 else np.uint32)
    want, carry = O.add(a, b, m)
    words, off = a.view(np.uint32).size, bits // 32
    (ba, pa), (bb, pb), (br, pr) = devmem.put(a, off), devmem.put(b, off), devmem.empty_words(words, off)
    dc = torch.full((n + 8,), 7, dtype=torch.uint8, device="cuda:0")
    s = torch.cuda.current_stream().cuda_stream
    ctx.add(pa, pb, pr, n, m, carry=dc.data_ptr(), limb_bits=bits, stream=s)
    torch.cuda.synchronize()
    assert np.array_equal(devmem.get(br, words, off, a.dtype), want)
    assert np.array_equal(dc.cpu().numpy()[:n], carry) and (dc.cpu().numpy()[n:] == 7).all()
    if bits == 64:
        ctx.add6(pa, pb, pr, n, m, stream=s)
        torch.cuda.synchronize()
        assert np.array_equal(devmem.get(br, words, off, a.dtype), O.add6(a, b, m))


@pytest.mark.parametrize("m", [49, 50, 51, 53, 54, 55, 96, 97, 99, 107, 108, 109])
def test_add_unaligned_rows_of_four_limbs_per_thread(ctx, devmem, m):
    # either side of the lengths that take consecutive limbs, in place and not
    n = 1300
    a, b = carry_stress(n, m, seed=m)
    want, carry = O.add(a, b, m)
    s = torch.cuda.current_stream().cuda_stream
    for inplace in (False, True):
        (ba, pa), (bb, pb), (br, pr) = devmem.put(a, 2), devmem.put(b, 2), devmem.empty_words(2 * n * m, 2)
        dc = torch.full((n + 8,), 7, dtype=torch.uint8, device="cuda:0")
        ctx.add(pa, pb, pa if inplace else pr, n, m, carry=dc.data_ptr(), stream=s)
        torch.cuda.synchronize()
        assert np.array_equal(devmem.get(ba if inplace else br, 2 * n * m, 2), want)
        assert np.array_equal(dc.cpu().numpy()[:n], carry) and (dc.cpu().numpy()[n:] == 7).all()
