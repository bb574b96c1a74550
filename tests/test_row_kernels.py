"""Row kernels at the row lengths where their pass plans change, against the oracle.

A row of C values runs log2 C - 2 butterfly stages and a product of 4-value polynomials;
how the stages split into passes depends on C and the radix.  n = 16 C on the tensor path
(16 rows), 32 C on the plain one, so these sizes cover C = 1 .. 4096 with every radix the
tuning accepts, one product and a batch, and coefficients of 0, 1 and q - 1 among random ones.
"""
import numpy as np
import pytest

import polymul
from oracle import oracle
from tests.helpers import from_ints, random_q, uniform_below

pytestmark = pytest.mark.gpu


def _inputs(n, q, limbs, count, seed):
    rng = np.random.default_rng(seed)
    x = [uniform_below(rng, q, n, limbs) for _ in range(2 * count)]
    edge = from_ints([0, 1, q - 1], limbs)
    for k, v in enumerate(x):
        v[k % n] = edge[2]
        v[n - 1] = edge[k % 3]
    x[0][:] = edge[2]  # every residue of the first product's a and b at its largest
    x[count][:] = edge[2]
    return np.stack(x[:count]), np.stack(x[count:])


@pytest.mark.parametrize("tensor", [True, False])
@pytest.mark.parametrize("n", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096, 8192, 16384, 32768, 65536])
def test_row_lengths_and_radices(cuda, n, tensor):
    torch = cuda
    q = random_q(np.random.default_rng(n), 130)
    count = 3 if n > 4096 else 9
    a, b = _inputs(n, q, 4, count, n + int(tensor))
    want = np.stack([oracle.rns_multiply(x, y, q) for x, y in zip(a, b)])
    da, db = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
    with polymul.Plan(n, q, 4, tensor=tensor) as p:
        for radix, persistent in [(16, 1), (8, 1), (4, 1), (8, 0), (4, 0)]:
            p.set_tuning(row_radix=radix, row_persistent=persistent)
            c = torch.zeros_like(da)
            p.multiply_batch(da.data_ptr(), db.data_ptr(), c.data_ptr(), count)
            one = torch.zeros_like(da[0])
            p.multiply(da.data_ptr(), db.data_ptr(), one.data_ptr())
            torch.cuda.synchronize()
            assert (c.cpu().numpy().view(np.uint64) == want).all(), (radix, persistent)
            assert (one.cpu().numpy().view(np.uint64) == want[0]).all(), (radix, persistent)


@pytest.mark.parametrize("tensor", [True, False])
@pytest.mark.parametrize("n,count", [(2, 4099), (16, 4099), (256, 1500)])
def test_large_default_groups_of_small_products(cuda, n, count, tensor):
    """More products than one default group of small rings holds: the same bits as groups of 100."""
    torch = cuda
    q = random_q(np.random.default_rng(n + count), 90)
    rng = np.random.default_rng(count)
    a, b = (uniform_below(rng, q, n * count, 2).reshape(count, n, 2) for _ in range(2))
    da, db = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
    with polymul.Plan(n, q, 2, tensor=tensor) as p:
        outs = []
        for group in (0, 100):
            p.set_tuning(group=group)
            c = torch.zeros_like(da)
            p.multiply_batch(da.data_ptr(), db.data_ptr(), c.data_ptr(), count)
            torch.cuda.synchronize()
            outs.append(c)
        assert torch.equal(outs[0], outs[1])
    for k in (0, 128, 4096 if count > 4096 else 1300, count - 1):
        assert (outs[0][k].cpu().numpy().view(np.uint64) == oracle.rns_multiply(a[k], b[k], q)).all()
