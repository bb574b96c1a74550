"""The conversion that folds column stages into its contraction, at the edges of its dispatch:
bases of 16 | 17 and 32 | 33 primes (three, two or one folded stage), rows too short for a
tile's columns (n = 128 .. 1024), launches just above the size it takes over at, and residue
planes that are 16- but not 32-byte aligned.  Against the per-prime-group conversion on
every product, and against the oracle on the first and last."""
import numpy as np
import pytest

import polymul
from oracle import oracle
from tests.helpers import from_ints, random_q, uniform_below

pytestmark = pytest.mark.gpu


def _bits_for(n, primes):
    """The widest q whose basis has `primes` primes at ring size n."""
    return max(b for b in range(2, 897) if len(polymul.basis(n, b)) == primes)


@pytest.mark.parametrize("n,primes,extra_limb", [
    (128, 16, 0), (256, 16, 0), (512, 16, 2), (1024, 16, 0), (1024, 17, 0), (2048, 16, 10),
    (256, 32, 0), (512, 32, 0), (1024, 32, 0), (1024, 33, 0), (4096, 32, 4), (4096, 33, 0),
    (256, 60, 0), (1024, 60, 0), (8192, 58, 0), (65536, 61, 0), (2048, 4, 0)])
def test_folded_conversion(cuda, n, primes, extra_limb):
    torch = cuda
    bits = _bits_for(n, primes)
    limbs = (bits + 127) // 128 * 2 + extra_limb
    limbs = min(limbs, 16)
    rng = np.random.default_rng(1000 * primes + n)
    q = random_q(rng, bits)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    count = 4 * sms * 128 // (2 * n) + 1  # the first count of more than 4 tiles of 128 an SM
    if n <= 1024:  # few distinct products, repeated
        base = [uniform_below(rng, q, n, limbs) for _ in range(6)]
        a = np.stack([base[k % 5] for k in range(count)])
        b = np.stack([base[(k + 1 + k // 5) % 6] for k in range(count)])
    else:
        a = np.stack([uniform_below(rng, q, n, limbs) for _ in range(count)])
        b = np.stack([uniform_below(rng, q, n, limbs) for _ in range(count)])
    a[0][:] = b[0][:] = from_ints([q - 1], limbs)[0]
    da, db = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
    with polymul.Plan(n, q, limbs, tensor=True) as p:
        assert p.primes == primes
        raw = torch.zeros(p.workspace_bytes * count + 64, dtype=torch.uint8, device="cuda")
        outs = []
        for whole, offset in [(1, 0), (1, 16), (0, 0)]:
            p.set_tuning(conv_whole_basis=whole, group=min(count, 256))
            c = torch.zeros_like(da)
            p.multiply_batch(da.data_ptr(), db.data_ptr(), c.data_ptr(), count, raw.data_ptr() + offset,
                             p.workspace_bytes * count)
            torch.cuda.synchronize()
            outs.append(c)
        assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[2])
        for k in (0, count - 1):
            got = outs[0][k].cpu().numpy().view(np.uint64)
            assert (got == oracle.rns_multiply(a[k], b[k], q)).all(), k
