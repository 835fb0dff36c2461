"""vf_apply_noalloc in a stream capture: the graph clears the completion counter
that its call keeps for every replay (a memset node ahead of the kernel), so a
replay does not depend on what an earlier one left, and replays between eager
calls (more of them than the ring of counters holds) give the same results.
Against a plain FP64 evaluation, 1e-13 of the largest value as elsewhere.  Both
kernel forms."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 300), (40, 17, 12)])
def test_replays_clear_their_counter(gpu, dims):
    import torch
    from cuda.bindings import runtime as rt
    from oracle import hex8
    from voxelsim_fea_b200 import _lib
    nx, ny, nz = dims
    nu = 0.29
    rng = np.random.default_rng(nx)
    nn, ne = (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz
    E = rng.uniform(0.5, 2.0, ne)
    mask = rng.integers(0, 8, nn).astype(np.uint8)
    free = ((mask[:, None] >> np.arange(3)) & 1).astype(bool).ravel()
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    E_d, m_d, u_d = dev(E), dev(mask), torch.empty(3 * nn, dtype=torch.float64, device="cuda")
    y, dot = torch.empty_like(u_d), torch.empty(1, dtype=torch.float64, device="cuda")

    def call():
        rc = _lib.load().vf_apply_noalloc(nx, ny, nz, nu, E_d.data_ptr(), m_d.data_ptr(), u_d.data_ptr(), y.data_ptr(),
                                          dot.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == _lib.VF_OK

    u_d.zero_()
    call()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    graph.instantiate()
    raw = rt.cudaGraph_t(graph.raw_cuda_graph())
    err, _, n = rt.cudaGraphGetNodes(raw, 0)
    assert err == rt.cudaError_t.cudaSuccess
    err, nodes, n = rt.cudaGraphGetNodes(raw, n)
    kinds = [rt.cudaGraphNodeGetType(k)[1] for k in nodes[:n]]
    assert kinds.count(rt.cudaGraphNodeType.cudaGraphNodeTypeMemset) == 1
    assert kinds.count(rt.cudaGraphNodeType.cudaGraphNodeTypeKernel) == 1
    edof, ke = hex8.build_edof(nx, ny, nz), hex8.hex8_ke(1.0, nu)
    for _ in range(3):
        u = rng.standard_normal(3 * nn)
        u_d.copy_(torch.from_numpy(u))
        ref = hex8.element_apply(u, E, edof, ke, 3 * nn) * free
        for k in range(70):
            y.fill_(float("nan"))
            dot.fill_(float("nan"))
            graph.replay() if k % 7 == 0 else call()
            if k % 7 < 2:
                scale = np.abs(ref).max()
                assert np.abs(y.cpu().numpy() - ref).max() <= 1e-13 * scale
                assert abs(dot.item() - float(u @ ref)) <= 1e-13 * np.abs(u).sum() * scale
