"""cuopo_crystal_pass_noalloc reports nothing from the device, so it must run
on one CTA: on a cluster a bounded wait could give up and leave the fields
half done with CUOPO_OK.  The launch is read from a captured graph (never
run)."""
import numpy as np
import pytest

import cuopo_b200 as cu
from cuopo_b200 import _lib
from tests.helpers import params_2eq, params_3eq

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def kernel_grids(call):
    """Grid sizes of the kernels that call(stream) launches."""
    from cuda.bindings import driver as dr

    def ok(r):
        assert r[0] == dr.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]
    stream = torch.cuda.Stream()
    ok(dr.cuStreamBeginCapture(stream.cuda_stream, dr.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED))
    call(stream.cuda_stream)
    graph = ok(dr.cuStreamEndCapture(stream.cuda_stream))
    count = ok(dr.cuGraphGetNodes(graph))[1]
    nodes = ok(dr.cuGraphGetNodes(graph, count))[0]
    grids = []
    for n in nodes:
        if ok(dr.cuGraphNodeGetType(n)) == dr.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            k = ok(dr.cuGraphKernelNodeGetParams(n))
            grids.append(k.gridDimX * k.gridDimY * k.gridDimZ)
    ok(dr.cuGraphDestroy(graph))
    return grids


@pytest.mark.parametrize("neq,n_t", [(q, n) for q in (2, 3) for n in (512, 1024, 2048, 4096, 8192)])
def test_noalloc_pass_runs_on_one_cta(neq, n_t):
    p = (params_2eq if neq == 2 else params_3eq)(n_t=n_t, n_z=4)
    A = [torch.zeros(n_t, dtype=torch.complex64, device="cuda") for _ in range(neq)]

    def call(stream):
        import ctypes as C
        _lib.check(cu.load().cuopo_crystal_pass_noalloc(C.byref(p), None, A[0].data_ptr(), A[1].data_ptr(),
                                                        A[2].data_ptr() if neq == 3 else None, stream))
    call(torch.cuda.current_stream().cuda_stream)   # kernels loaded, the array's address known
    torch.cuda.synchronize()
    assert kernel_grids(call) == [1]
