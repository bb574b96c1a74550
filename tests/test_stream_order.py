"""Products on a stream with other work before them.

The library's kernels may start while the kernel before them on the stream still runs and then wait
for it: behind a caller's kernel that lets its dependents start at once and outlasts the limit of
the kernels' bounded waits (1 s), in chains of products that feed one another, and in captured graphs,
whose buffers later calls must leave alone.  Against the oracle."""
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


def test_captured_batches_keep_the_plans_workspace(cuda):
    """A batch larger than the ones before it neither moves the buffer that captured graphs use nor
    needs a larger one during a capture."""
    torch = cuda
    n, bits, limbs = 1024, 200, 4
    rng = np.random.default_rng(5)
    q = random_q(rng, bits)
    few = [uniform_below(rng, q, n, limbs) for _ in range(5)]
    want = [[oracle.rns_multiply(x, y, q) for y in few] for x in few]
    pick = [(k % 5, (k // 5) % 5) for k in range(600)]
    da, db = (torch.from_numpy(np.stack([few[p[s]] for p in pick]).view(np.int64)).cuda() for s in (0, 1))
    with polymul.Plan(n, q, limbs) as p:
        def multiply(c):
            p.multiply_batch(da.data_ptr(), db.data_ptr(), c.data_ptr(), len(c),
                             stream=torch.cuda.current_stream().cuda_stream)

        outs = [torch.zeros((count, n, limbs), dtype=torch.int64, device="cuda") for count in (128, 600)]
        multiply(outs[0])
        torch.cuda.synchronize()
        graphs = []
        for c in outs:  # the second is larger than every batch before it
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                multiply(c)
            graphs.append(g)
            multiply(torch.zeros_like(outs[1]))
        for g, c in zip(graphs, outs):
            c.zero_()
            g.replay()
            torch.cuda.synchronize()
            got = c.cpu().numpy().view(np.uint64)
            assert all((got[k] == want[pick[k][0]][pick[k][1]]).all() for k in range(len(c)))


@pytest.mark.parametrize("n,bits,limbs,count", [
    (128, 300, 6, 2), (256, 868, 14, 1), (1024, 517, 9, 1), (4096, 868, 14, 2), (4096, 517, 9, 12),
    (1024, 868, 14, 40), (1024, 190, 3, 40), (16384, 400, 8, 1)])
def test_products_that_feed_one_another(cuda, n, bits, limbs, count):
    """Each product reads what the one before wrote, over two plans that share a workspace, with copies
    and another stream's work in between and no synchronisation; then the same captured."""
    torch = cuda
    rng = np.random.default_rng(n + bits + count)
    q = random_q(rng, bits)
    first = [uniform_below(rng, q, n, limbs) for _ in range(2)]
    a, b = (torch.from_numpy(np.stack([x] * count).view(np.int64)).cuda() for x in first)
    c, d = torch.zeros_like(a), torch.zeros_like(a)
    steps = 4
    side = torch.cuda.Stream()
    with polymul.Plan(n, q, limbs) as p1, polymul.Plan(n, q, limbs) as p2:
        ws = torch.zeros(p1.workspace_bytes * count, dtype=torch.uint8, device="cuda")

        def multiply(p, x, y, z):
            p.multiply_batch(x.data_ptr(), y.data_ptr(), z.data_ptr(), count, ws.data_ptr(), ws.numel(),
                             stream=torch.cuda.current_stream().cuda_stream)

        def chain(delay):
            x, y = a.clone(), b.clone()
            for _ in range(steps):
                multiply(p1, x, y, c)
                multiply(p2, c, x, d)
                here = torch.cuda.current_stream()
                side.wait_stream(here)
                with torch.cuda.stream(side):
                    if delay:
                        torch.cuda._sleep(200000)
                    x.copy_(d)
                here.wait_stream(side)
                multiply(p2, x, c, y)
            return y

        x, y = first
        for _ in range(steps):
            u = oracle.rns_multiply(x, y, q)
            x = oracle.rns_multiply(u, x, q)
            y = oracle.rns_multiply(x, u, q)
        for delay in (False, True):
            got = chain(delay).cpu().numpy().view(np.uint64)
            assert (got[0] == y).all() and (got[-1] == y).all()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = chain(False)
        for _ in range(2):
            c.zero_()
            graph.replay()
            got = out.cpu().numpy().view(np.uint64)
            assert (got[0] == y).all() and (got[-1] == y).all()
