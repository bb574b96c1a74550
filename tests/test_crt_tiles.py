"""The CRT kernel's tiles of 4 columns (launches of few products, bases of more than 48 primes): either
side of the launch size they stop at, rows of exactly one tile of 8, bases either side of 48 primes
and planes off a 16-byte boundary (read without tensor maps).  Against the oracle."""
import numpy as np
import pytest

import polymul
from oracle import oracle
from tests.helpers import from_ints, random_q, uniform_below

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bits,limbs", [
    (64, 868, 14), (128, 868, 14), (128, 720, 12), (256, 896, 14), (256, 715, 12), (512, 768, 12),
    (1024, 730, 16), (2048, 700, 12), (4096, 810, 13), (4096, 868, 14), (8192, 896, 14), (8192, 750, 15)])
def test_crt_tiles(cuda, n, bits, limbs):
    torch = cuda
    rng = np.random.default_rng(7 * n + bits)
    q = random_q(rng, bits)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    most = max(1, 4 * sms // (n // 16))  # products of the last launch in tiles of 4
    few = [uniform_below(rng, q, n, limbs) for _ in range(4)]
    few[0][:] = from_ints([q - 1], limbs)[0]
    for count in (1, most, most + 1):
        pick = [(k % 4, (k // 4 + k) % 4) for k in range(count)]
        da, db = (torch.from_numpy(np.stack([few[p[s]] for p in pick]).view(np.int64)).cuda() for s in (0, 1))
        with polymul.Plan(n, q, limbs) as p:
            raw = torch.zeros(p.workspace_bytes * count + 64, dtype=torch.uint8, device="cuda")
            p.set_tuning(group=min(count, 256))
            for offset in (0, 8) if limbs % 2 else (0,):
                c = torch.zeros_like(da)
                p.multiply_batch(da.data_ptr(), db.data_ptr(), c.data_ptr(), count, raw.data_ptr() + offset,
                                 p.workspace_bytes * count)
                torch.cuda.synchronize()
                got = c.cpu().numpy().view(np.uint64)
                for k in sorted({0, min(1, count - 1), count - 1}):
                    expect = oracle.rns_multiply(few[pick[k][0]], few[pick[k][1]], q)
                    assert (got[k] == expect).all(), (count, k, offset)
