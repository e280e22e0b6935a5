"""tff_system_kernel_launches against the kernel nodes of a captured evaluation: a small build, general
builds with the scan inside the key kernel and after it, slot parameters beside the neighbour search
and after it, planes and no PME, bonded terms. (A grid side of cuFFT's adds the kernels of that library,
which are not counted.)
"""
import numpy as np
import pytest
import torch
from cuda.bindings import runtime as cudart

from gpu_util import t

pytestmark = pytest.mark.gpu


def _kernel_nodes(call) -> int:
    call()  # outside the capture first: function attributes, module loading
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        call()
    graph = cudart.cudaGraph_t(g.raw_cuda_graph())
    err, _, n = cudart.cudaGraphGetNodes(graph)
    assert err == cudart.cudaError_t.cudaSuccess
    err, nodes, n = cudart.cudaGraphGetNodes(graph, n)
    assert err == cudart.cudaError_t.cudaSuccess
    kinds = [cudart.cudaGraphNodeGetType(v)[1] for v in nodes[:n]]
    return sum(k == cudart.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)


# 648, 1,026, 18,942 and 18,945 atoms (592 and 593 clusters), 99,000 atoms (32,768 keys)
@pytest.mark.parametrize("waters", [216, 342, 6314, 6315, 33000])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("grid", [0, 48])
def test_system(waters, dtype, grid):
    from torchff_b200.system import FixedChargeSystem
    from torchff_b200.water import serving_water_box

    wb = serving_water_box(waters, 1)
    wb.grid = grid
    sy = FixedChargeSystem.from_water_box(wb, dtype=dtype, flexible=waters == 342)
    x, box = t(wb.coords, dtype), t(wb.box, dtype)
    e, f = torch.empty(1, dtype=torch.float64, device="cuda"), torch.empty_like(x)
    assert _kernel_nodes(lambda: sy.evaluate_into(x, box, e, f)) == sy.kernel_launches()


def test_empty_system():
    from torchff_b200.system import FixedChargeSystem

    none = np.zeros(0)
    sy = FixedChargeSystem(none, none, none, None, 0.5, 3.0, 16, dtype=torch.float32)
    x = torch.zeros(0, 3, device="cuda")
    e, f = torch.empty(1, dtype=torch.float64, device="cuda"), torch.empty_like(x)
    box = t(np.eye(3), torch.float32)
    assert _kernel_nodes(lambda: sy.evaluate_into(x, box, e, f)) == sy.kernel_launches()
