"""blocks_per_sm of a flow map and of an FP64 batch: as many particles or threads in
flight as that number of blocks of 256 threads (of a batch: 128) holds at one lane a
particle, whatever the kernel's own block is."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class KernelNode(ctypes.Structure):
    """cudaKernelNodeParams"""
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("shared", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p)]


def _launches(call):
    """(blocks, threads of a block) of the kernels that call() launches"""
    import torch
    rt = ctypes.CDLL("libcudart.so.13")
    call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        call()
    graph, n = ctypes.c_void_p(g.raw_cuda_graph()), ctypes.c_size_t(16)
    nodes = (ctypes.c_void_p * 16)()
    assert rt.cudaGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    found = []
    for k in range(n.value):
        node, kind = ctypes.c_void_p(nodes[k]), ctypes.c_int()
        assert rt.cudaGraphNodeGetType(node, ctypes.byref(kind)) == 0
        if kind.value == 0:
            p = KernelNode()
            assert rt.cudaGraphKernelNodeGetParams(node, ctypes.byref(p)) == 0
            found.append((p.grid[0], p.block[0]))
    return found


@pytest.mark.parametrize("precision,lanes", [("fp64", 2), ("mixed", 1)])
@pytest.mark.parametrize("cap", [1, 2, 5])
def test_cap_is_the_same_amount_in_flight(nb, precision, lanes, cap):
    import torch
    dg, p, _ = nb.get_predefined_flow("double_gyre", int_direction=-1.0)
    x, y = (torch.linspace(0, b, n, dtype=torch.float64, device="cuda")
            for b, n in ((2.0, 1201), (1.0, 601)))
    out = torch.empty((1201, 601, 2), dtype=torch.float64, device="cuda")
    (blocks, threads), = _launches(lambda: nb.flowmap_grid_2D(
        dg, 0.0, -0.2, x, y, p, out=out, precision=precision, blocks_per_sm=cap))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert blocks * threads // lanes == sms * cap * 256
    whole = nb.flowmap_grid_2D(dg, 0.0, -0.2, x, y, p, precision=precision)
    assert torch.equal(out, whole)


@pytest.mark.parametrize("cap", [1, 3])
def test_cap_of_an_fp64_batch(nb, cap):
    import torch
    from numbacs_gb300.batch import Field, FTLEBatch
    dg, p, _ = nb.get_predefined_flow("double_gyre", int_direction=-1.0)
    x, y = np.linspace(0, 2, 601), np.linspace(0, 1, 301)
    b = FTLEBatch([Field(dg, 0.0, -0.2, x, y, p)], precision="fp64", blocks_per_sm=cap, graph=False)
    blocks, threads = _launches(b.launch)[1]    # after the counter's reset
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert blocks * threads // 2 == sms * cap * 128
