"""Performance cases of the batched big-integer library.

Each case is one call (or one list) that a program makes through the public
Python mirror of the C ABI (midint-arithmetic_gb300/midint.py): additions,
short chains, full products, low halves, the fused composite, ragged lists, and the calls on
host buffers.  Operands are uniform limbs with the worst-case rows that the
benchmark workloads add (carry chains for additions, all-ones operands for
products).  Results are whole numbers and compared bit for bit.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "midint-arithmetic_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import midint  # noqa: E402

_OPS = ("add", "chain", "mul", "mul_full", "mul_lo", "poly", "ragged", "host_mul", "gpu_multiply")


def listed():
    return [
        # (a + b) * b on a few short integers inside a larger program: launch and call latency
        {"name": "chain 1024-bit x256", "op": "chain", "n": 256, "limbs": 16, "bits": 64},
        # the plain batched addition of the benchmark, with carry-outs
        {"name": "add 4096-bit x65536", "op": "add", "n": 65536, "limbs": 64, "bits": 64},
        # additions wider than one thread block (multi-block carries), an odd length
        {"name": "add 64-Mbit x16", "op": "add", "n": 16, "limbs": 1048573, "bits": 64},
        # the headline batch: classical full products
        {"name": "mul_full 8192-bit x16384", "op": "mul_full", "n": 16384, "limbs": 128, "bits": 64},
        # a small batch of an uneven length through the size-picking product
        {"name": "mul 4352-bit x1500", "op": "mul", "n": 1500, "limbs": 68, "bits": 64},
        # long products: the size-picking call takes transforms
        {"name": "mul 65536-bit x1024", "op": "mul", "n": 1024, "limbs": 1024, "bits": 64},
        # products truncated to the operand length (the reference's product), odd u32 length
        {"name": "mul_lo 9632-bit x12000", "op": "mul_lo", "n": 12000, "limbs": 301, "bits": 32},
        # the fused composite (a^2+b)(b^2+b)+ab at the largest operand length
        {"name": "poly 131072-bit x512", "op": "poly", "n": 512, "limbs": 2048, "bits": 64},
        # the mixed list of the ragged benchmark, replayed as a captured graph
        {"name": "ragged 200000 ops", "op": "ragged", "n": 200000, "lo_bits": 256, "hi_bits": 65536, "graph": True},
        # one batch of a request loop: a short mixed list, launched directly
        {"name": "ragged 400 ops", "op": "ragged", "n": 400, "lo_bits": 512, "hi_bits": 32768, "graph": False},
        # the headline batch end to end between pinned host buffers
        {"name": "host_mul 8192-bit x16384", "op": "host_mul", "n": 16384, "limbs": 128, "bits": 64},
        # the reference's driver call on ordinary (pageable) host arrays
        {"name": "gpuMultiply 4096-bit x4096", "op": "gpu_multiply", "n": 4096, "limbs": 64, "bits": 64},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _seconds_per_product(limbs64):
    """A rough device time of one full product, to keep drawn cases below the
    cost of the listed ones."""
    return min(4.0 * limbs64 * limbs64 / 4e12, 1.2e-10 * limbs64 * max(4.0, math.log2(2.0 * limbs64)) / 1.3)


def draw(rng):
    op = rng.choice(_OPS + ("mul", "mul_full", "mul_lo"))
    if op == "ragged":
        n = _log_int(rng, 64, 150000)
        lo = rng.choice((256, 512, 1000))
        hi = rng.choice((8192, 32768, 65536))
        return {"op": op, "n": n, "lo_bits": lo, "hi_bits": hi, "graph": rng.random() < 0.5}
    if op == "add":
        bits = rng.choice((64, 64, 32))
        limbs = _log_int(rng, 4, 1 << 20) if bits == 64 else _log_int(rng, 7, 8191)
        total = _log_int(rng, 1 << 12, 1 << 22)
        n = max(4, min(1 << 20, total // limbs))
        return {"op": op, "n": n, "limbs": limbs, "bits": bits}
    if op == "chain":
        return {"op": op, "n": _log_int(rng, 64, 2048), "limbs": _log_int(rng, 8, 40), "bits": 64}
    bits = rng.choice((64, 32)) if op in ("mul_full", "mul_lo") else 64
    # mul_full and u32 products are always classical: their long operands are
    # rare in use and are drawn up to 24576 bits
    top = 384 if op == "mul_full" or bits == 32 else 1024 if op in ("host_mul", "gpu_multiply") else 2048
    if op == "host_mul":
        top = 256
    limbs64 = _log_int(rng, 4, top)
    limbs = limbs64 if bits == 64 else 2 * limbs64 - rng.randrange(2)
    one = _seconds_per_product(limbs64) * (4 if op == "poly" else 1)
    if op == "mul_full" or bits == 32:
        one = 4.0 * limbs64 * limbs64 / 4e12
    most = max(8, int(2.5e-4 / one))
    if op in ("host_mul", "gpu_multiply"):
        most = min(most, max(8, (1 << 21) // limbs64))
    n = _log_int(rng, 8, min(most, 1 << 18))
    return {"op": op, "n": n, "limbs": limbs, "bits": bits}


_ctx = None


def _context():
    """A program keeps one context per device for its whole life."""
    global _ctx
    if _ctx is None:
        _ctx = midint.Context(0)
    return _ctx


def _random(count, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randint(-(1 << 63), (1 << 63) - 1, (count,), dtype=torch.int64, device="cuda", generator=g)


def _operands(case, seed):
    """Two operand batches (n, limbs) as int64 (or int32) tensors on the GPU."""
    n, limbs, bits = case["n"], case["limbs"], case["bits"]
    words = n * limbs if bits == 64 else (n * limbs + 1) // 2
    a, b = _random(words, 2 * seed + 1), _random(words, 2 * seed + 2)
    if bits == 32:
        a, b = a.view(torch.int32)[: n * limbs].clone(), b.view(torch.int32)[: n * limbs].clone()
    a, b = a.view(n, limbs), b.view(n, limbs)
    first = seed % 8
    if case["op"] == "add":  # every 8th pair carries from end to end
        a[first::8] = -1
        b[first::8] = 0
        b[first::8, 0] = 1
    elif limbs * bits > 16384:  # every 16th pair of long operands: the largest digits
        a[first::16] = -1
        b[first::16] = -1
    return a, b


def _ragged(case, seed):
    """(ops, input limbs, output limbs): 40 % additions, 60 % products, both
    operand lengths log-uniform, packed in list order.  The seed sets the
    order; the operations are the case's own, so lists have one total size."""
    n = case["n"]
    rng = np.random.default_rng(n)
    lo, hi = math.log(case["lo_bits"]), math.log(case["hi_bits"])
    ops = np.zeros(n, midint.OP_DTYPE)
    kind = (rng.random(n) >= 0.4).astype(np.uint32)
    la = np.ceil(np.exp(rng.uniform(lo, hi, n)) / 64).astype(np.uint64)
    lb = np.ceil(np.exp(rng.uniform(lo, hi, n)) / 64).astype(np.uint64)
    order = np.random.default_rng(seed).permutation(n)
    kind, la, lb = kind[order], la[order], lb[order]
    ends = np.cumsum(la + lb)
    rlen = np.where(kind == midint.MI_OP_ADD, np.maximum(la, lb), la + lb)
    rends = np.cumsum(rlen)
    ops["kind"], ops["la"], ops["lb"] = kind, la, lb
    ops["a_off"] = ends - la - lb
    ops["b_off"] = ends - lb
    ops["r_off"] = rends - rlen
    return ops, int(ends[-1]), int(rends[-1])


def prepare(case, seed):
    s = {"case": case, "ctx": _context(), "stream": torch.cuda.current_stream().cuda_stream}
    op, n = case["op"], case["n"]
    if op == "ragged":
        ops, n_in, n_out = _ragged(case, seed)
        s["ops"] = torch.from_numpy(ops.view(np.uint8)).cuda()
        s["in"] = _random(n_in, seed)
        s["r"] = torch.zeros(n_out, dtype=torch.int64, device="cuda")
        s["carry"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
        s["bytes"] = midint.ragged_scratch_bytes(n)
        s["scratch"] = torch.empty(s["bytes"] // 4 + 1, dtype=torch.int32, device="cuda")
        if case["graph"]:
            s["graph"] = s["ctx"].ragged_graph(s["ops"], n, s["in"], s["r"], s["scratch"], s["bytes"],
                                               carry=s["carry"])
        return s
    a, b = _operands(case, seed)
    out = 2 if op in ("chain", "mul", "mul_full", "host_mul") else 1
    if op == "host_mul":
        s["a"], s["b"] = (torch.empty(x.shape, dtype=x.dtype, pin_memory=True).copy_(x) for x in (a, b))
        s["r"] = torch.zeros((n, out * case["limbs"]), dtype=torch.int64, pin_memory=True)
    elif op == "gpu_multiply":
        s["a"], s["b"] = (np.ascontiguousarray(x.cpu().numpy()).view(np.uint64).reshape(-1) for x in (a, b))
        s["r"] = np.zeros(n * case["limbs"], np.uint64)
    else:
        s["a"], s["b"] = a, b
        s["r"] = torch.empty((n, out * case["limbs"]), dtype=a.dtype, device="cuda")
        s["carry"] = torch.empty(n, dtype=torch.uint8, device="cuda") if op == "add" else None
        s["sum"] = torch.empty_like(a) if op == "chain" else None
    return s


def run(s):
    c, ctx, op = s["case"], s["ctx"], s["case"]["op"]
    if op == "ragged":
        if c["graph"]:
            s["graph"].launch(stream=s["stream"])
        else:
            ctx.ragged_run(s["ops"], c["n"], s["in"], s["r"], s["scratch"], s["bytes"], carry=s["carry"],
                           stream=s["stream"])
        return s["r"], s["carry"]
    if op == "host_mul":
        ctx.host_mul_full(s["a"], s["b"], s["r"], c["n"], c["limbs"])
        return s["r"]
    if op == "gpu_multiply":
        midint.gpuMultiply(midint.U64bits, c["limbs"], c["n"], s["a"], s["b"], s["r"])
        return s["r"].view(np.int64)
    if op == "add":
        ctx.add(s["a"], s["b"], s["r"], c["n"], c["limbs"], carry=s["carry"], limb_bits=c["bits"],
                stream=s["stream"])
        return s["r"], s["carry"]
    if op == "chain":
        ctx.add(s["a"], s["b"], s["sum"], c["n"], c["limbs"], stream=s["stream"])
        ctx.mul(s["sum"], s["b"], s["r"], c["n"], c["limbs"], stream=s["stream"])
        return s["sum"], s["r"]
    if op == "mul":
        ctx.mul(s["a"], s["b"], s["r"], c["n"], c["limbs"], stream=s["stream"])
    elif op == "mul_full":
        ctx.mul_full(s["a"], s["b"], s["r"], c["n"], c["limbs"], limb_bits=c["bits"], stream=s["stream"])
    elif op == "mul_lo":
        ctx.mul_lo(s["a"], s["b"], s["r"], c["n"], c["limbs"], limb_bits=c["bits"], stream=s["stream"])
    else:
        ctx.poly(s["a"], s["b"], s["r"], c["n"], c["limbs"], stream=s["stream"])
    return s["r"]


def _product_ops(w1, w2):
    """32-bit operations of a w1 x w2-word product: the quadratic count, or the
    reference's normalised 300 m lg m where that is lower."""
    m = max(w1, w2)
    return min(2.0 * w1 * w2, 300.0 * m * math.log2(max(2.0, m)))


def work(case):
    op, n = case["op"], case["n"]
    if op == "ragged":
        ops, n_in, n_out = _ragged(case, 1)
        mul = ops[ops["kind"] == midint.MI_OP_MUL]
        w1, w2 = 2.0 * mul["la"], 2.0 * mul["lb"]
        m = np.maximum(w1, w2)
        flops = float(np.minimum(2.0 * w1 * w2, 300.0 * m * np.log2(m)).sum())
        return {"bytes": 8.0 * (n_in + n_out) + 40.0 * n, "flops": flops + 2.0 * n_out}
    row = case["limbs"] * case["bits"] // 8
    words = case["limbs"] * case["bits"] // 32
    if op == "add":
        return {"bytes": n * (3.0 * row + 1), "flops": float(n) * words}
    full = op in ("mul", "mul_full", "host_mul")
    if op == "chain":  # a, b read, the sum and the product written
        return {"bytes": n * row * 5.0, "flops": n * (words + _product_ops(words, words))}
    flops = _product_ops(words, words) * {"poly": 2.0, "mul_lo": 0.5, "gpu_multiply": 0.5}.get(op, 1.0)
    return {"bytes": n * row * (4.0 if full else 3.0), "flops": n * flops}


def _ints(rows):
    """The integers of a (n, limbs) array, limb 0 least significant."""
    data = np.ascontiguousarray(rows)
    size = data.shape[1] * data.itemsize
    raw = data.tobytes()
    return [int.from_bytes(raw[i: i + size], "little") for i in range(0, len(raw), size)]


def _limbs(values, size):
    """Values (size bytes each, reduced) as one flat byte string."""
    mask = (1 << (8 * size)) - 1
    return b"".join((v & mask).to_bytes(size, "little") for v in values)


def exact(case, seed):
    op, n = case["op"], case["n"]
    if work(case)["flops"] > 2.5e9 and op != "poly" and case.get("limbs", 0) < 512:
        if op == "ragged" or n > 60000:
            return None  # minutes of big-integer products on the host
    if op == "ragged":
        ops, n_in, n_out = _ragged(case, seed)
        pool = _random(n_in, seed).cpu().numpy().tobytes()
        parts, carry = [], np.zeros(n, np.uint8)
        for i, o in enumerate(ops.tolist()):
            kind, la, lb, _, ao, bo, _ = o
            x = int.from_bytes(pool[8 * ao: 8 * (ao + la)], "little")
            y = int.from_bytes(pool[8 * bo: 8 * (bo + lb)], "little")
            if kind == midint.MI_OP_ADD:
                m = max(la, lb)
                carry[i] = (x + y) >> (64 * m)
                parts.append(_limbs([x + y], 8 * m))
            else:
                parts.append(_limbs([x * y], 8 * (la + lb)))
        return np.frombuffer(b"".join(parts), np.int64), carry
    a, b = (x.cpu().numpy() for x in _operands(case, seed))
    row = case["limbs"] * case["bits"] // 8
    word = np.int64 if case["bits"] == 64 else np.int32
    x, y = _ints(a), _ints(b)
    if op == "add":
        top = 8 * row
        s = [p + q for p, q in zip(x, y)]
        return (np.frombuffer(_limbs(s, row), word).reshape(n, -1),
                np.array([v >> top for v in s], np.uint8))
    if op == "chain":
        mask = (1 << (8 * row)) - 1
        s = [(p + q) & mask for p, q in zip(x, y)]
        v = [p * q for p, q in zip(s, y)]
        return (np.frombuffer(_limbs(s, row), word).reshape(n, -1),
                np.frombuffer(_limbs(v, 2 * row), word).reshape(n, -1))
    if op == "poly":
        v = [(p * p + q) * (q * q + q) + p * q for p, q in zip(x, y)]
    else:
        v = [p * q for p, q in zip(x, y)]
    out = row * 2 if op in ("mul", "mul_full", "host_mul") else row
    r = np.frombuffer(_limbs(v, out), word)
    return r if op == "gpu_multiply" else r.reshape(n, -1)
