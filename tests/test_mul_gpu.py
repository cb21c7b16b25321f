"""GPU classical multiplication vs the oracle, bit-exact, through the C ABI."""
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


def gpu_mul(ctx, devmem, a, b, m, full=True, limb_bits=64, offset=0):
    n = a.size // m
    in_words = a.view(np.uint32).size
    out_words = in_words * (2 if full else 1)
    ba, pa = devmem.put(a, offset)
    bb, pb = devmem.put(b, offset)
    br, pr = devmem.empty_words(out_words, offset)
    f = ctx.mul_full if full else ctx.mul_lo
    f(pa, pb, pr, n, m, limb_bits=limb_bits, stream=_stream())
    torch.cuda.synchronize()
    assert (br[offset + out_words:].cpu().numpy() == -1).all(), "result written past the batch"
    return devmem.get(br, out_words, offset, a.dtype)


U64_SIZES = [1, 2, 3, 4, 5, 8, 15, 16, 17, 31, 32, 33, 64, 100, 128, 129, 200, 256, 500, 512, 1000, 1024, 1025,
             1500, 2047, 2048]


@pytest.mark.parametrize("m", U64_SIZES)
@pytest.mark.parametrize("full", [True, False])
def test_mul_u64_matches_oracle(ctx, devmem, m, full):
    n = 37 if m <= 256 else 5
    a, b = carry_stress(n, m, seed=31 * m + full)
    assert np.array_equal(gpu_mul(ctx, devmem, a, b, m, full), O.mul(a, b, m, full))


@pytest.mark.parametrize("m", [1, 3, 7, 9, 15, 255, 257, 511, 2047, 4095])
@pytest.mark.parametrize("full", [True, False])
def test_mul_u32_odd_sizes(ctx, devmem, m, full):
    n = 11
    a, b = carry_stress(n, m, seed=m, dtype=np.uint32)
    assert np.array_equal(gpu_mul(ctx, devmem, a, b, m, full, limb_bits=32), O.mul(a, b, m, full))


@pytest.mark.parametrize("m", [4, 128, 1024])
def test_mul_unaligned(ctx, devmem, m):
    a, b = carry_stress(6, m, seed=m + 1)
    for off in (1, 2):
        got = gpu_mul(ctx, devmem, a.view(np.uint32), b.view(np.uint32), 2 * m, True, limb_bits=32, offset=off)
        assert np.array_equal(got.view(np.uint64), O.mul(a, b, m, True))


@pytest.mark.parametrize("m", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096])
def test_mul_matches_reference_fixtures(ctx, devmem, m):
    g = golden("ref_sweep.npz")
    assert np.array_equal(gpu_mul(ctx, devmem, g["a"], g["b"], m, full=False, limb_bits=32), g[f"mul_{m}"])
    f = golden("ref_full.npz")
    ha, hb = f[f"ha_{m}"], f[f"hb_{m}"]
    n, h = ha.size // m, m // 2
    lo_a = np.ascontiguousarray(ha.reshape(n, m)[:, :h]).ravel()
    lo_b = np.ascontiguousarray(hb.reshape(n, m)[:, :h]).ravel()
    assert np.array_equal(gpu_mul(ctx, devmem, lo_a, lo_b, h, full=True, limb_bits=32), f[f"hmul_{m}"])
    w = golden("ref_worst.npz")
    assert np.array_equal(gpu_mul(ctx, devmem, w[f"wa_{m}"], w[f"wa_{m}"], m, False, 32), w[f"wmul_{m}"])


def test_mul_all_ones_full(ctx, devmem):
    for m in (1, 64, 128, 1024, 2048):
        a = np.full(3 * m, 0xFFFFFFFFFFFFFFFF, np.uint64)
        assert np.array_equal(gpu_mul(ctx, devmem, a, a, m, True), O.mul(a, a, m, True))


def test_mul_config_shape(ctx, devmem):
    import workloads

    a, b = workloads.mul_pairs(n=16384, m=128)
    got = gpu_mul(ctx, devmem, a, b, 128, True)
    assert np.array_equal(got, O.batch_u64("mul", a, b, 128, threads=16))
    # the u32-limb variant of the same workload is the same bytes
    got32 = gpu_mul(ctx, devmem, a.view(np.uint32)[: 256 * 64], b.view(np.uint32)[: 256 * 64], 256, True, 32)
    assert np.array_equal(got32.view(np.uint64), got[: 64 * 256])


@pytest.mark.parametrize("m", [255, 256, 300, 384, 447, 448, 500, 512, 1000, 1024, 1500, 2047, 2048])
@pytest.mark.parametrize("lo_min", [1, 2049])
def test_mul_lo_u64_classical_and_ntt(ctx, devmem, m, lo_min):
    """mi_mul_lo_u64 with the low-half crossover forced to the NTT (1) and to
    the classical kernel (2049): the same low limbs as the oracle."""
    old = ctx.get_tuning(midint.TUNE_LO_NTT_MIN)
    ctx.set_tuning(midint.TUNE_LO_NTT_MIN, 0, lo_min)
    try:
        a, b = carry_stress(7, m, seed=5 * m + lo_min)
        assert np.array_equal(gpu_mul(ctx, devmem, a, b, m, full=False), O.mul(a, b, m, False))
        ones = np.full(3 * m, 0xFFFFFFFFFFFFFFFF, np.uint64)
        assert np.array_equal(gpu_mul(ctx, devmem, ones, ones, m, full=False), O.mul(ones, ones, m, False))
    finally:
        ctx.set_tuning(midint.TUNE_LO_NTT_MIN, 0, old)


def test_lo_ntt_min_knob(ctx):
    old = ctx.get_tuning(midint.TUNE_LO_NTT_MIN)
    for bad in (0, 2050):
        with pytest.raises(midint.MidintError):
            ctx.set_tuning(midint.TUNE_LO_NTT_MIN, 0, bad)
    assert ctx.get_tuning(midint.TUNE_LO_NTT_MIN) == old
    ctx.set_tuning(midint.TUNE_LO_NTT_MIN, 0, 2049)
    assert ctx.get_tuning(midint.TUNE_LO_NTT_MIN) == 2049
    ctx.set_tuning(midint.TUNE_LO_NTT_MIN, 0, old)


def test_compat_gpuMultiply(lib):
    g = golden("ref_sweep.npz")
    for m in (16, 256, 1024, 2048, 4096):  # the u64 form of the last three takes the NTT low half
        r = np.zeros_like(g["a"])
        midint.gpuMultiply(midint.U32bits, m, g["a"].size // m, g["a"], g["b"], r)
        assert np.array_equal(r, g[f"mul_{m}"])
        a64, b64 = g["a"].view(np.uint64), g["b"].view(np.uint64)
        r64 = np.zeros_like(a64)
        midint.gpuMultiply(midint.U64bits, m // 2, a64.size // (m // 2), a64, b64, r64)
        assert np.array_equal(r64.view(np.uint32), g[f"mul_{m}"])


def test_host_mul_full(ctx):
    a, b = carry_stress(700, 128, seed=12)
    r = np.zeros(700 * 256, np.uint64)
    ctx.host_mul_full(a, b, r, 700, 128)
    assert np.array_equal(r, O.mul(a, b, 128, True))


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("m", [1, 7, 8, 9, 23, 39, 41, 56, 72, 88, 104, 129, 136, 145, 160, 184, 193, 249, 255, 257,
                               264, 301, 320, 345, 520, 767, 1025, 1536])
def test_mul_lane_groups(ctx, devmem, m, full):
    # block counts whose groups are any number of lanes (5 to 32, several
    # products per warp, up to three rounds of anti-diagonals per lane), with a
    # few products and with enough for the rule to take more rounds
    big = 9000 if m <= 72 else 4000 if m <= 320 else 700
    a, b = carry_stress(big, m, seed=m, dtype=np.uint32)
    a[3 * m:4 * m] = b[3 * m:4 * m] = 0xFFFFFFFF
    want = O.mul(a, b, m, full)
    rl = 2 * m if full else m
    for n in (1, 37, 1216, big):
        if n <= big:
            got = gpu_mul(ctx, devmem, a[:n * m], b[:n * m], m, full, limb_bits=32, offset=n & 1)
            assert np.array_equal(got, want[:n * rl]), n


@pytest.mark.parametrize("m", [193, 200, 201, 208, 209, 223, 224, 225, 239, 240, 241, 255, 256])
def test_mul_karatsuba_batches(ctx, devmem, m):
    # 25..32 blocks in the batches that take one Karatsuba level (an odd count
    # leaves half a warp idle): halves of zeros, all ones and random values, equal
    # halves, halves that differ in one bit, in every combination of signs
    big = 4301
    rng = np.random.default_rng(m)
    half = 8 * ((m + 15) // 16)
    ops = []
    for _ in range(2):
        x = rng.integers(0, 2**32, (big, 2 * half), dtype=np.uint32)
        lo, hi = x[:, :half], x[:, half:]
        pick = rng.integers(0, 8, big)
        lo[pick == 0] = 0
        hi[pick == 1] = 0
        lo[pick == 2] = 0xFFFFFFFF
        hi[pick == 3] = 0xFFFFFFFF
        hi[pick == 4] = lo[pick == 4]
        hi[pick == 5] = lo[pick == 5] ^ np.uint32(1)
        x[pick == 6] = 0xFFFFFFFF
        ops.append(np.ascontiguousarray(x[:, :m]).reshape(-1))
    a, b = ops
    want = O.mul(a, b, m, True)
    for n, offset in ((big, 0), (big, 1), (1601, 0)):
        got = gpu_mul(ctx, devmem, a[:n * m], b[:n * m], m, True, limb_bits=32, offset=offset)
        assert np.array_equal(got, want[:n * 2 * m]), (n, offset)


@pytest.mark.parametrize("n", [1217, 1400, 1700, 2281, 2432, 3648])
@pytest.mark.parametrize("m,full", [(137, True), (177, True), (225, True), (137, False), (233, False), (301, False)])
def test_mul_balanced_launches(ctx, devmem, m, full, n):
    # batches whose launches keep their places to a multiple of four (a last
    # block or warp partly empty), on each of the forms the rule picks there
    a, b = carry_stress(n, m, seed=n + m, dtype=np.uint32)
    want = O.mul(a, b, m, full)
    for _ in range(2):
        assert np.array_equal(gpu_mul(ctx, devmem, a, b, m, full, limb_bits=32), want)


@pytest.mark.parametrize("m", [193, 255, 256, 383, 511])
def test_mul_lo_places(ctx, devmem, m):
    # low halves of 25 to 64 blocks in batches on either side of those whose
    # launches keep two places per SM (more than one and a half blocks, at most
    # two), two launches in a row
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per_block = 256 // (16 if m <= 256 else 32)
    for blocks in (sms * 3 // 2, sms * 3 // 2 + 1, 2 * sms, 2 * sms + 1):
        n = blocks * per_block - 1
        a, b = carry_stress(n, m, seed=blocks + m, dtype=np.uint32)
        want = O.mul(a, b, m, False)
        for _ in range(2):
            assert np.array_equal(gpu_mul(ctx, devmem, a, b, m, False, limb_bits=32), want), n


@pytest.fixture
def classical(ctx):
    """Full products on the classical kernels at every length and batch."""
    old = ctx.get_tuning(midint.TUNE_PLAIN_NTT_MIN)
    ctx.set_tuning(midint.TUNE_PLAIN_NTT_MIN, 0, 2049)
    yield ctx
    ctx.set_tuning(midint.TUNE_PLAIN_NTT_MIN, 0, old)


@pytest.mark.parametrize("m", [42, 64, 96, 100, 128, 129, 130, 160, 192, 200, 255, 256, 257, 258, 384, 500, 512, 513,
                               514, 768, 1000, 1024, 1025, 1026, 1500, 2047, 2048])
@pytest.mark.parametrize("offset", [0, 2])
def test_classical_full_products(classical, devmem, m, offset):
    # one warp to 512 threads per product (up to 128, 256, 512, 1024 and 2048
    # limbs), on rows that are 16-byte aligned (even lengths, no offset) or not:
    # lengths that small batches, and every batch from 129 limbs on, otherwise
    # take the transforms for
    n = 37 if m <= 256 else 9
    a, b = carry_stress(n, m, seed=m + offset)
    a[m:2 * m] = b[m:2 * m] = np.uint64(2**64 - 1)
    got = gpu_mul(classical, devmem, a, b, m, True, offset=offset)
    assert np.array_equal(got, O.mul(a, b, m, True))


@pytest.mark.parametrize("m", [128, 256, 512, 1024, 2048, 4096])
def test_classical_full_products_of_the_reference(classical, devmem, m):
    # the reference's own results: the full products behind its fixtures
    f = golden("ref_full.npz")
    if f"ha_{m}" not in f.files:
        pytest.skip("no fixture of this length")
    n, h = f[f"ha_{m}"].size // m, m // 2
    a, b = (np.ascontiguousarray(f[k].reshape(n, m)[:, :h]).ravel() for k in (f"ha_{m}", f"hb_{m}"))
    got = gpu_mul(classical, devmem, a.view(np.uint64), b.view(np.uint64), h // 2, True)
    assert np.array_equal(got.view(np.uint32), f[f"hmul_{m}"])
