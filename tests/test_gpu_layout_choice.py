"""The layout that a batch takes, read from its captured launch (threads per
CTA; the graph is never run).  Counts where several small CTAs per SM, or a
last wave that starts early, make the general kernel the faster one: us per
slice measured on the general kernel against the one-CTA spread layout."""
import numpy as np
import pytest

import cuopo_b200 as cu
from tests.helpers import params_2eq, params_3eq

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def kernel_blocks(call):
    """Threads per CTA of the kernels that call(stream) launches."""
    from cuda.bindings import driver as dr

    def ok(r):
        assert r[0] == dr.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]
    stream = torch.cuda.Stream()
    ok(dr.cuStreamBeginCapture(stream.cuda_stream, dr.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED))
    call(stream)
    graph = ok(dr.cuStreamEndCapture(stream.cuda_stream))
    count = ok(dr.cuGraphGetNodes(graph))[1]
    nodes = ok(dr.cuGraphGetNodes(graph, count))[0]
    blocks = [ok(dr.cuGraphKernelNodeGetParams(n)).blockDimX for n in nodes
              if ok(dr.cuGraphNodeGetType(n)) == dr.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL]
    ok(dr.cuGraphDestroy(graph))
    return blocks


@pytest.mark.parametrize("neq,n_t,prec,count,threads", [
    (3, 512, cu.F64, 1110, 32),     # 22.6 against 27.8
    (3, 1024, cu.F64, 200, 64),     # 11.7 against 12.7
    (3, 1024, cu.F64, 500, 64),     # 22.1 against 25.2
    (2, 1024, cu.F64, 200, 64),     # 11.2 against 11.8
    (2, 1024, cu.F32, 200, 256),    # the spread layout where it is the faster one: 5.5 against 6.7
    (3, 512, cu.F64, 339, 128),     # 10.0 against 11.2
    (2, 512, cu.F32, 260, 128)])    # 3.7 against 6.2
def test_batch_takes_the_faster_layout(neq, n_t, prec, count, threads):
    p = (params_2eq if neq == 2 else params_3eq)(n_t=n_t, n_z=2, regime=cu.CW)
    insts = [dict(n_t=n_t, ap0=p.ap0, Rs=0.97, delta=0.0, gdd=0.0, seed=0)] * count
    with cu.Batch(p, insts, precision=prec) as b:
        b.set_signal(np.zeros(b.total, np.complex64 if prec == cu.F32 else np.complex128))
        b.run(1, 0.0)
        torch.cuda.synchronize()

        def call(stream):
            b.step(1, 2, 0.0, stream=stream)
            b.wait(stream=stream)
        assert kernel_blocks(call) == [threads]
        torch.cuda.synchronize()
