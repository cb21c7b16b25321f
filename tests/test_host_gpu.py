"""Host-buffer calls (mi_host_*): every chunking of the copy/compute pipeline
and the zero-copy path on mapped pinned buffers give the oracle's results."""
from __future__ import annotations

import ctypes
import mmap

import numpy as np
import pytest
import torch

import midint
import oracle as O
from carry_data import carry_stress

pytestmark = pytest.mark.gpu


def _pinned(x: np.ndarray) -> torch.Tensor:
    t = torch.from_numpy(x.view(np.int64) if x.dtype == np.uint64 else x).pin_memory()
    return t


@pytest.fixture
def hctx(lib):
    c = midint.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("chunks", [1, 3, 8, 64])
@pytest.mark.parametrize("pinned", [False, True])
def test_host_mul_full_chunkings(hctx, chunks, pinned):
    n, m = 1000, 64
    a, b = carry_stress(n, m, seed=chunks)
    hctx.set_tuning(midint.TUNE_HOST_CHUNKS, 1, chunks)
    hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, 1, 0)
    want = O.mul(a, b, m, True)
    if pinned:
        pa, pb = _pinned(a), _pinned(b)
        pr = torch.zeros(2 * n * m, dtype=torch.int64).pin_memory()
        hctx.host_mul_full(pa, pb, pr, n, m)
        got = pr.numpy().view(np.uint64)
    else:
        got = np.zeros(2 * n * m, np.uint64)
        hctx.host_mul_full(a, b, got, n, m)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("chunks", [1, 5, 16])
def test_host_add_chunkings(hctx, chunks):
    n, m = 3001, 33
    a, b = carry_stress(n, m, seed=chunks + 100)
    hctx.set_tuning(midint.TUNE_HOST_CHUNKS, 0, chunks)
    hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, 0, 0)
    r = np.zeros(n * m, np.uint64)
    c = np.zeros(n, np.uint8)
    hctx.host_add(a, b, r, c, n, m)
    ra, ca = O.add(a, b, m)
    assert np.array_equal(r, ra) and np.array_equal(c, ca)


def test_zero_copy_on_pinned_buffers(hctx):
    hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, 0, 1)
    hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, 1, 1)
    n, m = 777, 128
    a, b = carry_stress(n, m, seed=9)
    pa, pb = _pinned(a), _pinned(b)
    pr = torch.zeros(2 * n * m, dtype=torch.int64).pin_memory()
    hctx.host_mul_full(pa, pb, pr, n, m)
    assert np.array_equal(pr.numpy().view(np.uint64), O.mul(a, b, m, True))
    na, ma = 2049, 64
    a, b = carry_stress(na, ma, seed=10)
    pa, pb = _pinned(a), _pinned(b)
    pr = torch.zeros(na * ma, dtype=torch.int64).pin_memory()
    pc = torch.zeros(na, dtype=torch.uint8).pin_memory()
    hctx.host_add(pa, pb, pr, pc, na, ma)
    ra, ca = O.add(a, b, ma)
    assert np.array_equal(pr.numpy().view(np.uint64), ra) and np.array_equal(pc.numpy(), ca)
    # pageable buffers fall back to the copy pipeline
    r = np.zeros(na * ma, np.uint64)
    c = np.zeros(na, np.uint8)
    hctx.host_add(a, b, r, c, na, ma)
    assert np.array_equal(r, ra) and np.array_equal(c, ca)


@pytest.mark.parametrize("chunks", [1, 3, 8])
@pytest.mark.parametrize("pinned", [False, True])
def test_copied_operands_with_results_in_place(hctx, chunks, pinned):
    """Mode 3: operands copied in by chunks, results written in place."""
    for cls in (0, 1):
        hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, cls, 3)
        hctx.set_tuning(midint.TUNE_HOST_CHUNKS, cls, chunks)
    n, m = 515, 64
    a, b = carry_stress(n, m, seed=chunks + 31)
    if pinned:
        pr = torch.zeros(2 * n * m, dtype=torch.int64).pin_memory()
        hctx.host_mul_full(_pinned(a), _pinned(b), pr, n, m)
        got = pr.numpy().view(np.uint64)
    else:  # pageable results: the copy pipeline
        got = np.zeros(2 * n * m, np.uint64)
        hctx.host_mul_full(a, b, got, n, m)
    assert np.array_equal(got, O.mul(a, b, m, True))
    ra, ca = O.add(a, b, m)
    if pinned:
        pr = torch.zeros(n * m, dtype=torch.int64).pin_memory()
        pc = torch.zeros(n, dtype=torch.uint8).pin_memory()
        hctx.host_add(a, b, pr, pc, n, m)
        r, c = pr.numpy().view(np.uint64), pc.numpy()
    else:
        r, c = np.zeros(n * m, np.uint64), np.zeros(n, np.uint8)
        hctx.host_add(a, b, r, c, n, m)
    assert np.array_equal(r, ra) and np.array_equal(c, ca)
    # a wide addition with its results in place
    mw = 5000
    aw, bw = carry_stress(3, mw, seed=4)
    rw = torch.zeros(3 * mw, dtype=torch.int64).pin_memory()
    cw = torch.zeros(3, dtype=torch.uint8).pin_memory()
    hctx.host_add(aw, bw, rw, cw, 3, mw)
    raw, caw = O.add(aw, bw, mw)
    assert np.array_equal(rw.numpy().view(np.uint64), raw) and np.array_equal(cw.numpy(), caw)


@pytest.mark.parametrize("blocks", [1, 2, 3])
def test_zero_copy_with_capped_occupancy(hctx, blocks):
    """Mode 1 with the product kernel held to 1..3 resident blocks per SM."""
    hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, 1, 1)
    hctx.set_tuning(midint.TUNE_HOST_ZC_BLOCKS, 1, blocks)
    assert hctx.get_tuning(midint.TUNE_HOST_ZC_BLOCKS, 1) == blocks
    for n, m in ((1500, 128), (999, 64), (37, 5), (64, 512)):
        a, b = carry_stress(n, m, seed=blocks * 100 + m)
        pa, pb = _pinned(a), _pinned(b)
        pr = torch.zeros(2 * n * m, dtype=torch.int64).pin_memory()
        hctx.host_mul_full(pa, pb, pr, n, m)
        assert np.array_equal(pr.numpy().view(np.uint64), O.mul(a, b, m, True))
    hctx.set_tuning(midint.TUNE_HOST_ZC_BLOCKS, 1, 0)


@pytest.mark.parametrize("m", [64, 128])
def test_zero_copy_strides_over_a_large_batch(hctx, m):
    """Mode 1 on a batch larger than the capped grid (32 blocks per SM of
    256 threads): each group reads its next instance's operands while it
    multiplies the current one, over several rounds and a ragged last one."""
    hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, 1, 1)
    hctx.set_tuning(midint.TUNE_HOST_ZC_BLOCKS, 1, 2)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per_block = 256 // (m // 4)  # instances of one 256-thread block (groups of m/4 threads)
    n = sms * 32 * per_block + 777
    a, b = carry_stress(n, m, seed=m + 5)
    pa, pb = _pinned(a), _pinned(b)
    pr = torch.zeros(2 * n * m, dtype=torch.int64).pin_memory()
    hctx.host_mul_full(pa, pb, pr, n, m)
    assert np.array_equal(pr.numpy().view(np.uint64), O.mul(a, b, m, True))
    hctx.set_tuning(midint.TUNE_HOST_ZC_BLOCKS, 1, 0)


@pytest.mark.parametrize("chunks", [1, 3, 8])
@pytest.mark.parametrize("pinned_out", [False, True])
def test_zero_copy_reads_with_copied_results(hctx, chunks, pinned_out):
    """Mode 2: operands read in place, results copied out in chunks."""
    for cls in (0, 1):
        hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, cls, 2)
        hctx.set_tuning(midint.TUNE_HOST_CHUNKS, cls, chunks)
    n, m = 513, 64
    a, b = carry_stress(n, m, seed=chunks + 7)
    pa, pb = _pinned(a), _pinned(b)
    if pinned_out:
        pr = torch.zeros(2 * n * m, dtype=torch.int64).pin_memory()
        hctx.host_mul_full(pa, pb, pr, n, m)
        got = pr.numpy().view(np.uint64)
    else:
        got = np.zeros(2 * n * m, np.uint64)
        hctx.host_mul_full(pa, pb, got, n, m)
    assert np.array_equal(got, O.mul(a, b, m, True))
    r = np.zeros(n * m, np.uint64)
    c = np.zeros(n, np.uint8)
    hctx.host_add(pa, pb, r, c, n, m)
    ra, ca = O.add(a, b, m)
    assert np.array_equal(r, ra) and np.array_equal(c, ca)
    # a wide addition in this mode keeps its launches on one stream
    mw = 5000
    aw, bw = carry_stress(3, mw, seed=2)
    rw = np.zeros(3 * mw, np.uint64)
    cw = np.zeros(3, np.uint8)
    hctx.host_add(_pinned(aw), _pinned(bw), rw, cw, 3, mw)
    raw, caw = O.add(aw, bw, mw)
    assert np.array_equal(rw, raw) and np.array_equal(cw, caw)


def test_host_tuning_knobs_are_checked(hctx):
    with pytest.raises(midint.MidintError):
        hctx.set_tuning(midint.TUNE_HOST_CHUNKS, 0, 0)
    with pytest.raises(midint.MidintError):
        hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, 0, 4)
    with pytest.raises(midint.MidintError):
        hctx.set_tuning(midint.TUNE_HOST_CHUNKS, 2, 4)
    with pytest.raises(midint.MidintError):
        hctx.set_tuning(midint.TUNE_HOST_ZC_BLOCKS, 1, 4)
    with pytest.raises(midint.MidintError):
        hctx.set_tuning(midint.TUNE_HOST_ZC_BLOCKS, 2, 1)
    hctx.set_tuning(midint.TUNE_HOST_CHUNKS, 1, 5)
    assert hctx.get_tuning(midint.TUNE_HOST_CHUNKS, 1) == 5


@pytest.mark.parametrize("m", [320, 512, 2048])
def test_compat_gpuMultiply_ntt_low_half_on_pinned_buffers(lib, m):
    """The u64 gpuMultiply wrapper takes the NTT low half from 320 limbs on;
    on mapped pinned buffers its kernel reads and writes them in place (the
    tuned zero-copy mode of products), on pageable ones through copies."""
    n = 40
    a, b = carry_stress(n, m, seed=m + 3)
    want = O.mul(a, b, m, False)
    pa, pb = _pinned(a), _pinned(b)
    pr = torch.zeros(n * m, dtype=torch.int64).pin_memory()
    midint.check(lib.mi_compat_gpuMultiply_u64(n, m, pa.data_ptr(), pb.data_ptr(), pr.data_ptr()))
    assert np.array_equal(pr.numpy().view(np.uint64), want)
    r = np.zeros(n * m, np.uint64)
    midint.gpuMultiply(midint.U64bits, m, n, a, b, r)
    assert np.array_equal(r, want)


def test_contexts_on_several_host_threads(lib):
    """Host threads with their own contexts and different zero-copy occupancy
    caps (different shared-memory requests of the same product kernel) call
    at once; every result is the oracle's."""
    import threading

    n, m = 600, 128
    a, b = carry_stress(n, m, seed=404)
    want = O.mul(a, b, m, True)
    pa, pb = _pinned(a), _pinned(b)
    outs = [torch.zeros(2 * n * m, dtype=torch.int64).pin_memory() for _ in range(4)]
    ctxs = [midint.Context(0) for _ in range(4)]
    errors = []
    start = threading.Barrier(4)

    def run(i):
        try:
            ctxs[i].set_tuning(midint.TUNE_HOST_ZERO_COPY, 1, 1)
            ctxs[i].set_tuning(midint.TUNE_HOST_ZC_BLOCKS, 1, i)
            start.wait()
            for _ in range(3):
                ctxs[i].host_mul_full(pa, pb, outs[i], n, m)
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in ctxs:
        c.close()
    assert not errors, errors
    for o in outs:
        assert np.array_equal(o.numpy().view(np.uint64), want)


def test_calib_host_link(ctx):
    # SM-driven streaming over mapped pinned memory: plausible rates, and
    # sizes that are not a multiple of 32 bytes refused before any launch
    nb = 8 << 20
    src = torch.empty(nb, dtype=torch.uint8).pin_memory()
    dst = torch.empty(nb, dtype=torch.uint8).pin_memory()
    r, w, b = midint.calib_host_link(src, dst, nb)
    assert 1.0 < r < 5000.0 and 1.0 < w < 5000.0 and 1.0 < b < 10000.0
    with pytest.raises(midint.MidintError) as e:
        midint.calib_host_link(src, dst, nb - 16)
    assert e.value.status == midint.MI_EINVAL


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("n,m", [(1, 1), (9, 5), (513, 64), (1500, 128), (40, 700), (30000, 33), (400, 2048)])
def test_ordinary_arrays(hctx, mode, n, m):
    """Ordinary (pageable) arrays, which modes 1 and 2 use in place up to
    32 MiB where the GPU can: results that were never written before, operands
    at the edge of a page, a result over an operand, mixed with pinned ones."""
    for cls in (0, 1):
        hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, cls, mode)
    a, b = carry_stress(n, m, seed=n + m)
    full, (ra, ca) = O.mul(a, b, m, True), O.add(a, b, m)
    r = np.empty(2 * n * m + 2, np.uint64)
    r[0] = r[-1] = 77
    hctx.host_mul_full(a, b, r[1:-1], n, m)
    assert np.array_equal(r[1:-1], full) and r[0] == r[-1] == 77
    s, c = np.empty(n * m, np.uint64), np.empty(n + 8, np.uint8)
    c[n:] = 7
    hctx.host_add(a, b, s, c, n, m)
    assert np.array_equal(s, ra) and np.array_equal(c[:n], ca) and (c[n:] == 7).all()
    pr = torch.zeros(2 * n * m, dtype=torch.int64).pin_memory()
    hctx.host_mul_full(a, _pinned(b), pr, n, m)
    assert np.array_equal(pr.numpy().view(np.uint64), full)
    over = a.copy()
    hctx.host_add(over, b, over, None, n, m)   # in place: as the device call
    assert np.array_equal(over, ra)
    # at four bytes past a multiple of eight: copied, whatever the mode
    odd = np.zeros(4 * n * m + 4, np.uint32)[1:]
    hctx.host_mul_full(a, b, odd[:4 * n * m], n, m)
    assert np.array_equal(odd[:4 * n * m].copy().view(np.uint64), full)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("n,m", [(700, 1), (700, 3), (700, 5), (300, 13), (300, 127), (9, 2047), (5, 2049), (5, 4095)])
def test_host_add_on_odd_lengths(hctx, mode, n, m):
    # rows that allow no 16-byte access, read over the host link or staged
    hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, 0, mode)
    a, b = carry_stress(n, m, seed=n + m)
    want, carry = O.add(a, b, m)
    r = torch.zeros(n * m + 1, dtype=torch.int64).pin_memory()
    c = torch.full((n + 8,), 7, dtype=torch.uint8).pin_memory()
    hctx.host_add(_pinned(a), _pinned(b), r, c, n, m)
    assert np.array_equal(r.numpy().view(np.uint64)[:-1], want) and r[-1] == 0
    assert np.array_equal(c.numpy()[:n], carry) and (c.numpy()[n:] == 7).all()


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("n,m", [(700, 1), (700, 9), (700, 11), (300, 13), (300, 17), (9, 2049), (5, 4095), (5, 4097),
                                 (5, 8191)])
def test_gpuAdd_u32_on_odd_lengths(hctx, pinned, n, m):
    a, b = carry_stress(n, m, seed=n + m, dtype=np.uint32)
    keep = [_pinned(x.view(np.int32)) if pinned else x for x in (a, b, np.zeros(n * m, np.uint32))]
    a2, b2, r = [k.numpy().view(np.uint32) if pinned else k for k in keep]
    midint.gpuAdd(midint.U32bits, m, n, a2, b2, r)
    assert np.array_equal(r, O.add(a, b, m)[0])


@pytest.mark.parametrize("n", [1, 31, 33, 1000])
@pytest.mark.parametrize("m", [1, 2, 3, 7, 8, 9, 11, 16, 17, 23, 24, 31, 32, 33, 40, 95, 96, 120, 129, 255, 256, 301, 600])
def test_gpuMultiply_runs_of_rows(m, n):
    """Low halves of u32 limbs on pinned buffers: one to 32 products per warp, the
    last warp's partly empty, whole 16-byte words or not, from words past the last
    row that must not be read into a product."""
    n = n if m < 256 else min(n, 100)
    a, b = carry_stress(n, m, seed=n + m, dtype=np.uint32)
    pad = np.full(64, 0xFFFFFFFF, np.uint32)
    keep = [_pinned(np.concatenate([x, pad]).view(np.int32)) for x in (a, b, np.zeros(n * m, np.uint32))]
    a2, b2, r = [k.numpy().view(np.uint32)[:n * m] for k in keep]
    midint.gpuMultiply(midint.U32bits, m, n, a2, b2, r)
    assert np.array_equal(r, O.mul(a, b, m, False))
    assert (keep[2].numpy()[n * m:] == -1).all()


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("m", [287, 288, 301, 320, 512, 514])
def test_gpuMultiply_either_side_of_the_link_rule(m, pinned):
    # few products (transforms from 288 limbs on) and more than six per SM,
    # which stay classical over the host link up to 512 limbs of even length
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    a, b = carry_stress(6 * sms + 1, m, seed=m)
    want = O.mul(a, b, m, False)
    for n in (3, 6 * sms, 6 * sms + 1):
        keep = [_pinned(x) if pinned else x for x in (a[:n * m].copy(), b[:n * m].copy(), np.zeros(n * m, np.uint64))]
        a2, b2, r = [k.numpy().view(np.uint64) if pinned else k for k in keep]
        midint.gpuMultiply(midint.U64bits, m, n, a2, b2, r)
        assert np.array_equal(r, want[:n * m]), n


def _in_place_device():
    """Whether the GPU walks the host's page tables (device attributes 88 and 100)."""
    cudart = ctypes.CDLL("libcudart.so.13")
    v = ctypes.c_int()
    for attr in (88, 100):
        if cudart.cudaDeviceGetAttribute(ctypes.byref(v), attr, 0) != 0 or not v.value:
            return False
    return True


def _mapped(x: np.ndarray, prot: int, at_end: bool):
    """x in an anonymous mapping of its own, at its start or so that it ends
    exactly with its last page, which an inaccessible page follows."""
    page = mmap.PAGESIZE
    size = -(-x.nbytes // page) * page
    mm = mmap.mmap(-1, size + page)
    base = ctypes.addressof(ctypes.c_char.from_buffer(mm))
    off = size - x.nbytes if at_end else 0
    view = np.frombuffer(mm, x.dtype, x.size, off)
    view[:] = x
    libc = ctypes.CDLL(None, use_errno=True)
    libc.mprotect.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int]
    assert libc.mprotect(base + size, page, 0) == 0
    assert libc.mprotect(base, size, prot) == 0
    return view, (mm, libc, base, size + page)


def _release(keep):
    mm, libc, base, size = keep
    assert libc.mprotect(base, size, mmap.PROT_READ | mmap.PROT_WRITE) == 0


def _free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("at_end", [False, True])
@pytest.mark.parametrize("n,m", [(1000, 64), (333, 129)])
def test_ordinary_memory_is_used_in_place(hctx, at_end, n, m):
    # operands that may only be read and that end at an inaccessible page, a result
    # in fresh pages; the staging buffers of the copies are never allocated
    for cls in (0, 1):
        hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, cls, 1)
    a, b = carry_stress(n, m, seed=n)
    rw = mmap.PROT_READ | mmap.PROT_WRITE
    (va, ka), (vb, kb) = (_mapped(x, mmap.PROT_READ, at_end) for x in (a, b))
    vr, kr = _mapped(np.zeros(2 * n * m, np.uint64), rw, at_end)
    before = _free_bytes()
    hctx.host_mul_full(va, vb, vr, n, m)
    after = _free_bytes()
    assert np.array_equal(vr, O.mul(a, b, m, True))
    vs, ks = _mapped(np.zeros(n * m, np.uint64), rw, at_end)
    hctx.host_add(va, vb, vs, None, n, m)
    assert np.array_equal(vs, O.add(a, b, m)[0])
    if _in_place_device():
        assert before - after < n * m * 8, "staged: the copies' buffers were allocated"
    for k in (ka, kb, kr, ks):
        _release(k)


def test_operands_in_a_private_file_mapping(hctx, tmp_path):
    # pages of a file, and a result over the 32 MiB that are used in place
    for cls in (0, 1):
        hctx.set_tuning(midint.TUNE_HOST_ZERO_COPY, cls, 1)
    for n, m in ((700, 64), (20000, 64)):
        a, b = carry_stress(n, m, seed=n)
        path = tmp_path / f"operand{n}"
        path.write_bytes(a.tobytes())
        fa = np.memmap(path, np.uint64, "r")
        r = np.zeros(2 * n * m, np.uint64)
        hctx.host_mul_full(fa, b, r, n, m)
        assert np.array_equal(r, O.mul(a, b, m, True))


def test_populating_a_result_that_may_not_be_written_fails():
    # what sends such a call back to the copies, as any buffer that cannot be used
    # in place (the copies would then meet the same protection, as before)
    libc = ctypes.CDLL(None, use_errno=True)
    libc.madvise.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int]
    view, keep = _mapped(np.zeros(4096, np.uint64), mmap.PROT_READ, False)
    populate_read, populate_write = 22, 23
    assert libc.madvise(keep[2], mmap.PAGESIZE, populate_read) == 0
    assert libc.madvise(keep[2], mmap.PAGESIZE, populate_write) != 0
    _release(keep)


@pytest.mark.parametrize("m,n", [(5, 157286), (5, 157287), (8, 98303), (8, 98305), (11, 23831), (11, 23833), (24, 10925),
                                 (95, 2761), (96, 2731)])
def test_gpuMultiply_runs_of_rows_from_their_size_on(m, n):
    """Either side of the operand size (1 MB, 3 MB for rows of one block) from
    which a warp reads its rows as one run."""
    a, b = carry_stress(n, m, seed=n + m, dtype=np.uint32)
    keep = [_pinned(x.view(np.int32)) for x in (a, b, np.zeros(n * m, np.uint32))]
    a2, b2, r = [k.numpy().view(np.uint32) for k in keep]
    midint.gpuMultiply(midint.U32bits, m, n, a2, b2, r)
    assert np.array_equal(r, O.mul(a, b, m, False))
