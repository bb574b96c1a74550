"""pm_kernel_launch_count over an uneven batch: one kernel per conversion class (folded stages), ring
size and CRT width."""
import numpy as np
import pytest

import polymul
from tests.helpers import random_q

pytestmark = pytest.mark.gpu


def test_uneven_batch_counts_every_launch(cuda):
    torch = cuda
    # 660 tiles of 128 coefficients; three, two and one folded stage (14 primes, 28, and 59 or rows of 16)
    sizes = [(32768, 868), (8192, 400), (1024, 200), (256, 200)]
    rng = np.random.default_rng(3)
    batch = polymul.Batch([n for n, _ in sizes], [random_q(rng, bits) for _, bits in sizes], 14)
    before = polymul.launch_count()
    batch.run(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    batch.check_errors()
    conversions, ring_sizes, widths = 3, 4, 3
    assert polymul.launch_count() - before == conversions + ring_sizes + widths
