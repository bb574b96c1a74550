"""What a user of this library has it compute, as timed cases over its public entry points.

A case is one call (or one batch) of exact products c = a * b mod (X^n + 1, q):

  product       Plan.multiply             one product on device buffers
  batch         Plan.multiply_batch       many products of one (n, q) on device buffers
  host_product  Plan.multiply_host        one product on host arrays (the drop-in's call)
  host_batch    Plan.multiply_host_batch  many products on pinned host arrays
  uneven        Batch.run                 products of different n and q, copied in and out on the device

Ring sizes, widths and layouts are those of the tests and the benchmark: n = 256 .. 65536, q of
100 .. 896 bits, coefficients stored in the limbs q needs or padded to the 14 of the FHERMA layout.
Plans keep their defaults, as a program that only creates one and multiplies has them.
"""
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "fherma-polymul-baseline_b200"))
import polymul  # noqa: E402

FHERMA_Q = (1 << 868) - 11993087
BATCH_WORDS = 128 * 32768 * 14      # u64 words of one of a, b, c in the largest device batch
HOST_WORDS = 32 * 16384 * 14        # the same for host arrays
UNEVEN = 32                         # products of the listed uneven batch


def listed():
    def case(name, kind, n, bits, limbs, count=1):
        return {"name": name, "kind": kind, "n": n, "bits": bits, "limbs": limbs, "count": count}

    return [
        # the smallest call: one product of a small ring, where launches and latency count
        case("product_1k", "product", 1024, 868, 14),
        # an ordinary ring, one product at a time (an interactive caller with data on the GPU)
        case("product_4k", "product", 4096, 868, 14),
        # the FHERMA point, one product at a time
        case("product_32k", "product", 32768, 868, 14),
        # many small products of a narrow modulus (a batched low-depth scheme)
        case("batch_1k_narrow", "batch", 1024, 200, 4, 500),
        # a modulus that needs an odd number of limbs, stored unpadded: half of all widths do
        case("batch_4k_odd", "batch", 4096, 517, 9, 60),
        # ordinary batches of ordinary rings
        case("batch_8k", "batch", 8192, 868, 14, 100),
        case("batch_16k", "batch", 16384, 640, 10, 51),
        # the headline: a launch group of FHERMA-sized products
        case("batch_32k", "batch", 32768, 868, 14, 128),
        # the largest ring and width
        case("batch_64k", "batch", 65536, 896, 14, 24),
        # the drop-in's call: pageable arrays in, one product, pageable array out
        case("host_product_32k", "host_product", 32768, 868, 14),
        # products streamed from pinned host memory
        case("host_batch_16k", "host_batch", 16384, 868, 14, 32),
        # products of different rings and moduli, n 1024 .. 65536, 200 .. 868 bits
        {"name": "uneven_batch", "kind": "uneven", "count": UNEVEN, "limbs": 14, "mix": 4},
    ]


def draw(rng):
    kind = rng.choices(["product", "batch", "host_product", "host_batch", "uneven"], [5, 9, 2, 2, 2])[0]
    if kind == "uneven":
        return {"kind": kind, "count": rng.randint(4, UNEVEN), "limbs": 14, "mix": rng.randrange(1 << 20)}
    n = 1 << rng.randint(8, 16)
    bits = rng.randint(100, 896)
    limbs = 14 if rng.random() < 0.4 else (bits + 63) // 64
    count = 1
    if kind in ("batch", "host_batch"):
        most = min(1024, (BATCH_WORDS if kind == "batch" else HOST_WORDS) // (n * limbs))
        count = int(round(2 * (most / 2) ** rng.random()))
    return {"kind": kind, "n": n, "bits": bits, "limbs": limbs, "count": count}


def _modulus(bits, rng):
    return rng.getrandbits(bits) | (1 << (bits - 1)) | 1


def _uneven_sizes(case):
    """The batch's (n, bits), which are the case's own: n log-uniform, widths uniform."""
    rng = random.Random(case["mix"])
    return [(1 << rng.randint(10, 16), rng.randint(200, 868)) for _ in range(case["count"])]


def _q(case):
    # a program's modulus is fixed; its coefficients vary from call to call
    if case["bits"] == 868:
        return FHERMA_Q
    return _modulus(case["bits"], random.Random(1000003 * case["bits"] + case["n"]))


def _uniform(q, rows, limbs, gen):
    """rows coefficients below q as (rows, limbs) int64 words on the generator's device: the top
    62 bits of each uniform below q's, the bits under them uniform (q of more than 62 bits)."""
    dev = gen.device
    shift = q.bit_length() - 62
    w, b = divmod(shift, 64)
    x = torch.zeros((rows, limbs), dtype=torch.int64, device=dev)
    info = torch.iinfo(torch.int64)
    low = torch.randint(info.min, info.max, (rows, w + 1), dtype=torch.int64, device=dev, generator=gen)
    top = torch.randint(0, q >> shift, (rows,), dtype=torch.int64, device=dev, generator=gen)
    x[:, :w] = low[:, :w]
    x[:, w] = (top << b) | (low[:, w] & ((1 << b) - 1)) if b else top
    if b > 2:
        x[:, w + 1] = top >> (64 - b)
    return x


def _inputs(case, seed, device):
    """Seeded a and b of every product: (count, n, limbs) int64, or the packed words of an uneven batch."""
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    if case["kind"] == "uneven":
        rng = random.Random(case["mix"] + 1)
        qs = [_modulus(bits, rng) for _, bits in _uneven_sizes(case)]
        ab = [torch.cat([_uniform(q, n, case["limbs"], gen).flatten() for (n, _), q in zip(_uneven_sizes(case), qs)])
              for _ in range(2)]
        return qs, ab[0], ab[1]
    q = _q(case)
    shape = (case["count"], case["n"], case["limbs"])
    rows = case["count"] * case["n"]
    return q, _uniform(q, rows, case["limbs"], gen).view(shape), _uniform(q, rows, case["limbs"], gen).view(shape)


def prepare(case, seed):
    kind = case["kind"]
    q, a, b = _inputs(case, seed, "cuda")
    if kind == "uneven":
        batch = polymul.Batch([n for n, _ in _uneven_sizes(case)], q, case["limbs"])
        return {"kind": kind, "batch": batch, "a": a, "b": b, "c": torch.empty_like(a)}
    if kind.startswith("host"):
        a, b = a.cpu(), b.cpu()
        if kind == "host_batch":
            a, b = a.pin_memory(), b.pin_memory()
            c = torch.zeros_like(a).pin_memory()
        else:
            a, b = (x[0].numpy().view(np.uint64) for x in (a, b))
            c = np.zeros_like(a)
    else:
        c = torch.empty_like(a)
    plan = polymul.Plan(case["n"], q, coef_limbs=case["limbs"])
    return {"kind": kind, "plan": plan, "count": case["count"], "a": a, "b": b, "c": c}


def run(state):
    kind, a, b, c = (state[k] for k in ("kind", "a", "b", "c"))
    if kind == "host_product":
        return state["plan"].multiply_host(a, b, out=c).view(np.int64)
    if kind == "host_batch":
        state["plan"].multiply_host_batch_ptr(a.data_ptr(), b.data_ptr(), c.data_ptr(), state["count"])
        return c
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "uneven":
        batch = state["batch"]
        batch.copy_in(a.data_ptr(), b.data_ptr(), stream)
        batch.run(stream)
        batch.copy_out(c.data_ptr(), stream)
    elif kind == "batch":
        state["plan"].multiply_batch(a.data_ptr(), b.data_ptr(), c.data_ptr(), state["count"], stream=stream)
    else:
        state["plan"].multiply(a.data_ptr(), b.data_ptr(), c.data_ptr(), stream=stream)
    return c


def _shapes(case):
    """(n, bits) of every product of a case."""
    return _uneven_sizes(case) if case["kind"] == "uneven" else [(case["n"], case["bits"])] * case["count"]


def work(case):
    """a and b read once and c written once; the operations (multiply, add, subtract) of three
    negacyclic transforms of size n over the 30-bit residues the exact product needs."""
    nbytes = flops = 0
    for n, bits in _shapes(case):
        logn = n.bit_length() - 1
        residues = -(-(2 * bits + 2 + logn) // 30)
        nbytes += 3 * n * case["limbs"] * 8
        flops += residues * (3 * 3 * (n // 2) * logn + n)
    return {"bytes": nbytes, "flops": flops}


def _negacyclic(a, b, n, q):
    """a * b mod (X^n + 1, q), (n, limbs) int64 words in and out, by one multiplication of the
    polynomials packed into integers."""
    limbs = a.shape[1]
    slot = (2 * q.bit_length() + n.bit_length() + 7) // 8
    pad = max(0, slot - 8 * limbs)

    def packed(x):
        rows = x.tobytes()
        return int.from_bytes(b"".join(rows[8 * limbs * i:8 * limbs * i + min(slot, 8 * limbs)] + bytes(pad)
                                       for i in range(n)), "little")

    prod = (packed(a) * packed(b)).to_bytes(2 * n * slot, "little")
    term = [int.from_bytes(prod[slot * i:slot * (i + 1)], "little") for i in range(2 * n)]
    out = b"".join(((term[i] - term[n + i]) % q).to_bytes(8 * limbs, "little") for i in range(n))
    return np.frombuffer(out, dtype=np.int64).reshape(n, limbs)


def exact(case, seed):
    """Python's own integers, where they take seconds: the residues are whole numbers."""
    # one product of 1024 coefficients of 868 bits takes 0.2 s, and time grows as size^1.585
    seconds = sum(0.25 * (n * bits / (1024 * 868)) ** 1.585 for n, bits in _shapes(case))
    if seconds > 8:
        return None
    q, a, b = _inputs(case, seed, "cuda")
    a, b = a.cpu().numpy(), b.cpu().numpy()
    if case["kind"] == "uneven":
        limbs, at, parts = case["limbs"], 0, []
        for (n, _), qz in zip(_uneven_sizes(case), q):
            words = slice(at, at + n * limbs)
            parts.append(_negacyclic(a[words].reshape(n, limbs), b[words].reshape(n, limbs), n, qz).flatten())
            at += n * limbs
        return torch.from_numpy(np.concatenate(parts))
    c = np.stack([_negacyclic(x, y, case["n"], q) for x, y in zip(a, b)])
    return torch.from_numpy(c[0].copy() if case["kind"] == "host_product" else c)
