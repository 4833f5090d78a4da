"""Short products captured with their tables in place: the graph holds no memory
of its own, so that it may have several instances at once and be part of another
graph."""
import ctypes

import numpy as np
import pytest

from gpu_util import to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb", [(300, 300), (383, 383), (5000, 100), (20000, 40), (100000, 300)])
def test_instances_and_child_graph(oracle, na, nb):
    import torch
    import natural_number_gb300 as nn
    cu = ctypes.CDLL("libcuda.so.1")
    void = ctypes.c_void_p
    a, b = limbs(na, na), limbs(nb + 3, nb)
    want = [oracle.mul(a, b), oracle.sqr(b)]
    stream = torch.cuda.Stream()
    st = void(stream.cuda_stream)
    with torch.cuda.stream(stream):
        da, db = to_dev(a), to_dev(b)
        out = [torch.empty(k, dtype=torch.uint64, device="cuda") for k in (na + nb, 2 * nb)]
        ctx = nn.Context(0)

        def work():
            ctx.mul_device(out[0], da, db)
            ctx.sqr_device(out[1], db)

        def check():
            stream.synchronize()
            for o, w in zip(out, want):
                got = to_host(o)
                assert np.array_equal(got[: w.size], w) and not got[w.size:].any()
                o.view(torch.int64).zero_()

        ctx.mul_device(torch.empty(2 * na, dtype=torch.uint64, device="cuda"), da, da)  # tables for any of these
        work()
        check()
        graph, outer, node = void(), void(), void()
        assert cu.cuStreamBeginCapture_v2(st, 2) == 0  # relaxed
        work()
        assert cu.cuStreamEndCapture(st, ctypes.byref(graph)) == 0
        assert cu.cuGraphCreate(ctypes.byref(outer), 0) == 0
        assert cu.cuGraphAddChildGraphNode(ctypes.byref(node), outer, None, ctypes.c_size_t(0), graph) == 0
        instances = []
        for g in (graph, graph, outer):
            e = void()
            assert cu.cuGraphInstantiateWithFlags(ctypes.byref(e), g, ctypes.c_ulonglong(0)) == 0
            instances.append(e)
        for e in instances:
            assert cu.cuGraphLaunch(e, st) == 0
            check()
        for e in instances:
            cu.cuGraphExecDestroy(e)
        cu.cuGraphDestroy(outer)
        cu.cuGraphDestroy(graph)
        ctx.close()
