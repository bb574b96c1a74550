"""Uneven batches either side of the number of tiles from which they convert by the folding kernel:
one small product, several classes of basis, and the last batch below the line and the first above it.
Against the oracle, before and after the batch autotuner."""
import numpy as np
import pytest

import polymul
from oracle import oracle
from tests.helpers import from_ints, random_q, uniform_below

pytestmark = pytest.mark.gpu


def _line(torch):
    """Products of n = 1024 (16 tiles of 128 coefficients) up to three tiles an SM."""
    return 3 * torch.cuda.get_device_properties(0).multi_processor_count // 16


@pytest.mark.parametrize("sizes,more", [
    ([(256, 868)], None), ([(256, 60), (256, 240), (512, 470), (1024, 896)], None),
    ([(2048, 100), (8192, 868), (256, 500)], None), ([], 0), ([], 1)])
def test_small_batches(cuda, sizes, more):
    if more is not None:
        sizes = [(1024, (200, 400, 868)[k % 3]) for k in range(_line(cuda) + more)]
    rng = np.random.default_rng(len(sizes))
    qs = [random_q(rng, bits) for _, bits in sizes]
    a, b = ([uniform_below(rng, q, n, 14) for (n, _), q in zip(sizes, qs)] for _ in range(2))
    a[0][:] = b[0][:] = from_ints([qs[0] - 1], 14)[0]
    want = [oracle.rns_multiply(x, y, q) for x, y, q in zip(a, b, qs)]
    with polymul.Batch([n for n, _ in sizes], qs) as batch:
        for _ in range(2):
            got = batch.multiply_host(a, b)
            batch.check_errors()
            assert all((x == y).all() for x, y in zip(got, want))
            batch.autotune(reps=1)
