"""What apollo_dg_rhs_noalloc puts on a stream (B200): on aligned arrays one
clear of the call's state and one stage kernel, by the nodes of a captured graph."""
import ctypes as C

import numpy as np
import pytest

from apollo_b200 import NodalDG2d, problems

pytestmark = pytest.mark.gpu


def test_two_nodes():
    torch = pytest.importorskip("torch")
    rt = pytest.importorskip("cuda.bindings.runtime")
    p = problems.euler_vortex(n=9, N=3)
    s = NodalDG2d(p.N, p.cfl, p.equation, p.eq_params, p.mesh)
    x, y = s.node_coords()
    u = torch.from_numpy(np.ascontiguousarray(p.ic(x, y))).cuda()
    out = torch.empty_like(u)
    stream = torch.cuda.Stream()

    def call():
        s._check(s.lib.apollo_dg_rhs_noalloc(s.h, 0.0, 0.0, C.c_void_p(u.data_ptr()), C.c_void_p(out.data_ptr()), None,
                                             C.c_void_p(stream.cuda_stream)))

    torch.cuda.synchronize()
    call()  # the first call looks the static array up
    torch.cuda.synchronize()
    ref = out.clone()
    out.zero_()
    torch.cuda.synchronize()
    assert rt.cudaStreamBeginCapture(stream.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)[0] == 0
    call()
    err, graph = rt.cudaStreamEndCapture(stream.cuda_stream)
    assert err == 0
    kinds = [rt.cudaGraphNodeGetType(n)[1] for n in rt.cudaGraphGetNodes(graph, 16)[1][:rt.cudaGraphGetNodes(graph)[2]]]
    t = rt.cudaGraphNodeType
    assert sorted(int(k) for k in kinds) == sorted([int(t.cudaGraphNodeTypeMemset), int(t.cudaGraphNodeTypeKernel)])
    err, g = rt.cudaGraphInstantiate(graph, 0)
    assert err == 0 and rt.cudaGraphLaunch(g, stream.cuda_stream)[0] == 0
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
    rt.cudaGraphExecDestroy(g)
    rt.cudaGraphDestroy(graph)
