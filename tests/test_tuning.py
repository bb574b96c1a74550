"""Launch shapes as asked for (the grids that a captured product's kernels have under each tuning), and
the autotuner's choice among those that differ."""
import ctypes

import numpy as np
import pytest

import polymul
from tests.helpers import random_q

pytestmark = pytest.mark.gpu


class KernelNode(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("shared", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def _crt_grid(torch, plan, count, limbs):
    """CTAs of the CRT kernel in a captured batch of `count` products."""
    a = torch.zeros((count, plan.n, limbs), dtype=torch.int64, device="cuda")
    c, ws = torch.zeros_like(a), torch.zeros(plan.workspace_bytes * count, dtype=torch.uint8, device="cuda")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        plan.multiply_batch(a.data_ptr(), a.data_ptr(), c.data_ptr(), count, ws.data_ptr(), ws.numel(),
                            stream=torch.cuda.current_stream().cuda_stream)
    cu = ctypes.CDLL("libcuda.so.1")
    number = ctypes.c_size_t(64)
    nodes = (ctypes.c_void_p * 64)()
    assert cu.cuGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), nodes, ctypes.byref(number)) == 0
    grids = []
    for node in nodes[:number.value]:
        k, name = KernelNode(), ctypes.c_char_p()
        assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(k)) == 0
        assert cu.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(k.func)) == 0
        if b"k3t_crt" in name.value:
            grids.append(k.grid[0])
    assert len(grids) == 1
    return grids[0]


@pytest.mark.parametrize("bits,limbs,fit", [(200, 4, 3), (384, 6, 3), (385, 8, 2), (868, 14, 2)])
def test_crt_ctas_per_sm_is_what_was_asked_for(cuda, bits, limbs, fit):
    torch = cuda
    q = random_q(np.random.default_rng(bits), bits)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n, count = 2048, 60  # 960 tiles of 8 columns, more than 4 x 148
    with polymul.Plan(n, q, limbs) as p:
        assert _crt_grid(torch, p, count, limbs) == fit * sms
        for k in (1, 2, 3, 4):
            p.set_tuning(crt_ctas_per_sm=k, group=count)
            assert _crt_grid(torch, p, count, limbs) == k * sms
        p.set_tuning(group=count)  # the rest as in an untuned plan
        assert _crt_grid(torch, p, count, limbs) == fit * sms
        chosen = p.autotune()
        p.set_tuning(crt_ctas_per_sm=chosen["crt_ctas_per_sm"], group=count)
        assert _crt_grid(torch, p, count, limbs) == chosen["crt_ctas_per_sm"] * sms


def test_autotuner_weighs_the_default_group(cuda):
    """Launch shapes that only repeat the default's are not picked: with the default group of 585 small
    products (one launch instead of five, half the time), with a default of 128, and with the
    conversion of rows without tensor maps, which has one form."""
    rng = np.random.default_rng(9)
    with polymul.Plan(1024, random_q(rng, 200), 4) as p:
        default = p.batch_workspace_size(5000)
        assert p.autotune()["group"] == 0
        assert p.batch_workspace_size(5000) == default
    with polymul.Plan(16384, random_q(rng, 517), 9) as p:
        chosen = p.autotune()
        assert chosen["group"] != 128 and chosen["conv_whole_basis"] == 1
