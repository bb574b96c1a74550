"""Products on a stream with other work before them.

The library's kernels may start while the kernel before them on the stream still runs and then wait
for it.  Here that kernel is the caller's own: it lets its dependents start at once and runs for
longer than the limit of the kernels' bounded waits (1 s), which must not run against it.
Both conversion kernels, with tensor maps and without, against the oracle."""
import numpy as np
import pytest

from oracle import oracle
import polymul
from tests.helpers import random_q, uniform_below

pytestmark = pytest.mark.gpu

# releases its dependents, then runs for `ms` milliseconds (or 10 million steps at the most)
EARLY = r"""
extern "C" __global__ void early(int ms, unsigned long long* ran) {
    unsigned long long t0, t;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    int steps = 0;
    do {
        __nanosleep(1000);
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    } while (t - t0 < ms * 1000000ull && ++steps < 10000000);
    *ran = t - t0;
}
"""


@pytest.mark.parametrize("n,bits,limbs,count", [
    (1024, 868, 14, 1), (1024, 517, 9, 1), (1024, 868, 14, 40), (1024, 190, 3, 40)])
def test_bounded_waits_start_after_the_previous_kernel(cuda, n, bits, limbs, count):
    torch = cuda
    rng = np.random.default_rng(n + bits + count)
    q = random_q(rng, bits)
    a, b = uniform_below(rng, q, n, limbs), uniform_below(rng, q, n, limbs)
    da, db = (torch.from_numpy(np.stack([x] * count).view(np.int64)).cuda() for x in (a, b))
    early = torch.cuda._compile_kernel(EARLY, "early")
    ran = torch.zeros(1, dtype=torch.int64, device="cuda")
    with polymul.Plan(n, q, limbs) as p:
        ws = torch.zeros(p.workspace_bytes * count, dtype=torch.uint8, device="cuda")
        c = torch.zeros_like(da)
        stream = torch.cuda.current_stream().cuda_stream
        torch.cuda.synchronize()
        early(grid=(1, 1, 1), block=(1, 1, 1), args=[1500, ran])
        p.multiply_batch(da.data_ptr(), db.data_ptr(), c.data_ptr(), count, ws.data_ptr(), ws.numel(), stream=stream)
        torch.cuda.synchronize()
        assert ran.item() > 1.2e9  # it did outlast the limit
        got = c.cpu().numpy().view(np.uint64)
        want = oracle.rns_multiply(a, b, q)
        for k in (0, count - 1):
            assert (got[k] == want).all()
        # the plan's error word: no wait gave up
        assert (p.multiply_host(a, b) == want).all()
