"""Which form vf_apply_noalloc takes, read from the kernel node of a captured call
(32 x 8 threads: marching, 256 x 1: gather).  Grids whose tiles of 31 x 7 columns
are mostly empty, or whose march is one long chain, take the gather form, which is
2 to 20 times faster there; grids that fill tiles take the marching form."""

import pytest

pytestmark = pytest.mark.gpu

GATHER = [(7, 7, 8000), (3, 9, 2000), (1, 200, 200), (3, 40, 3000), (2, 100, 400), (1, 1, 100000), (200000, 1, 1),
          (2000000, 1, 1), (1, 62, 3000), (3, 3, 40000), (2, 1000, 300)]
MARCH = [(1, 1, 1), (48, 24, 24), (16, 16, 16), (61, 43, 37), (30, 6, 1000), (10, 3, 200), (251, 127, 129),
         (10000, 10, 10), (1000, 1000, 1), (32, 8, 2000), (15, 7, 4000)]


@pytest.mark.parametrize("dims,form", [(d, (256, 1)) for d in GATHER] + [(d, (32, 8)) for d in MARCH])
def test_form(gpu, dims, form):
    import torch
    from cuda.bindings import driver as cu
    from voxelsim_fea_b200 import _lib
    nx, ny, nz = dims
    nn, ne = (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz
    E = torch.ones(ne, dtype=torch.float64, device="cuda")
    mask = torch.full((nn,), 7, dtype=torch.uint8, device="cuda")
    u = torch.zeros(3 * nn, dtype=torch.float64, device="cuda")
    y, dot = torch.empty_like(u), torch.empty(1, dtype=torch.float64, device="cuda")

    def call():
        assert _lib.load().vf_apply_noalloc(nx, ny, nz, 0.3, E.data_ptr(), mask.data_ptr(), u.data_ptr(), y.data_ptr(),
                                            dot.data_ptr(), torch.cuda.current_stream().cuda_stream) == _lib.VF_OK

    call()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw = cu.CUgraph(graph.raw_cuda_graph())
    n = cu.cuGraphGetNodes(raw, 0)[2]
    nodes = cu.cuGraphGetNodes(raw, n)[1][:n]
    kernels = [k for k in nodes if cu.cuGraphNodeGetType(k)[1] == cu.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL]
    assert len(kernels) == 1
    err, params = cu.cuGraphKernelNodeGetParams(kernels[0])
    assert err == cu.CUresult.CUDA_SUCCESS
    assert (params.blockDimX, params.blockDimY) == form
