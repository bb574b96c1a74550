"""Plans over an odd number of limbs with no path asked for: the tensor path with coefficient
rows loaded without tensor maps.  Small launches and ones of more than four tiles an SM, one
to three folded stages, buffers on 8-byte boundaries (accepted as on the plain method),
the host calls; bit-exact against the plain method and the oracle."""
import numpy as np
import pytest

import polymul
from oracle import oracle
from tests.helpers import from_ints, random_q, uniform_below

pytestmark = pytest.mark.gpu


def _product_inputs(n, bits, limbs, count, seed):
    rng = np.random.default_rng(seed)
    q = random_q(rng, bits)
    base = [uniform_below(rng, q, n, limbs) for _ in range(min(2 * count, 7))]
    a = np.stack([base[k % len(base)] for k in range(count)])
    b = np.stack([base[(k * 3 + 1) % len(base)] for k in range(count)])
    a[0][:] = b[0][:] = from_ints([q - 1], limbs)[0]
    a[-1][n - 1] = 0
    return q, a, b


@pytest.mark.parametrize("n,bits,limbs,count", [
    (128, 300, 5, 3), (256, 63, 1, 3), (256, 831, 13, 5), (512, 130, 3, 40), (1024, 190, 3, 40), (1024, 446, 7, 300),
    (1024, 190, 3, 300), (4096, 517, 9, 2), (4096, 517, 9, 12), (8192, 300, 5, 6), (16384, 700, 11, 3),
    (32768, 831, 13, 2), (65536, 150, 3, 1), (2048, 200, 13, 24)])
@pytest.mark.parametrize("shift", [0, 1])
def test_odd_limbs_match_plain_method(cuda, n, bits, limbs, count, shift):
    torch = cuda
    q, a, b = _product_inputs(n, bits, limbs, count, n + bits + count)
    words = count * n * limbs

    def at(x):  # the array at `shift` words past a 16-byte boundary
        buf = torch.zeros(words + 2, dtype=torch.int64, device="cuda")
        if x is not None:
            buf[shift:shift + words] = torch.from_numpy(x.view(np.int64).reshape(-1)).cuda()
        return buf, buf.data_ptr() + 8 * shift

    (da, pa), (db, pb) = at(a), at(b)
    outs = []
    for tensor in (None, False):
        with polymul.Plan(n, q, limbs, tensor=tensor) as p:
            assert p.tensor == (tensor is None and n >= 256)
            ws = torch.zeros(p.workspace_bytes * count // 8 + 2, dtype=torch.int64, device="cuda")
            dc, pc = at(None)
            p.multiply_batch(pa, pb, pc, count, ws.data_ptr() + 8 * shift, p.workspace_bytes * count)
            torch.cuda.synchronize()
            assert not dc[:shift].any() and not dc[shift + words:].any()
            outs.append(dc[shift:shift + words].cpu().numpy().view(np.uint64).reshape(a.shape))
    assert (outs[0] == outs[1]).all()
    for k in {0, count - 1}:
        assert (outs[0][k] == oracle.rns_multiply(a[k], b[k], q)).all()


@pytest.mark.parametrize("n,bits,limbs", [(256, 63, 1), (4096, 517, 9), (32768, 831, 13)])
def test_odd_limbs_host_calls(cuda, n, bits, limbs):
    q, a, b = _product_inputs(n, bits, limbs, 5, n)
    with polymul.Plan(n, q, limbs) as p:
        assert p.tensor
        got = p.multiply_host_batch(a, b)
        for k in range(5):
            assert (got[k] == p.multiply_host(a[k], b[k])).all()
        p.set_tuning(conv_whole_basis=0)  # no per-group form without tensor maps: the same kernels
        assert (p.multiply_host(a[1], b[1]) == got[1]).all()
    for k in (0, 4):
        assert (got[k] == oracle.rns_multiply(a[k], b[k], q)).all()
