"""A captured render keeps its image when the context has rendered in another
storage form since: the volumes that the FAST schedule reads in F16 and those
that exact filtering reads in U8 are buffers of their own."""
import ctypes as C

import numpy as np
import pytest

from pedalsky_b200 import capi, scenes
from pedalsky_b200.capi import call
from pedalsky_b200.subsystem import subsystem_for_scene

from . import _gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,then", [(capi.STORAGE_F16, capi.STORAGE_U8), (capi.STORAGE_U8, capi.STORAGE_F16)])
def test_captured_render_survives_a_change_of_storage(oracle_noise, first, then):
    torch = _gpu.torch_cuda()
    s = scenes.precision_1080p(96, 54, storage=first, schedule=capi.SCHED_FAST, filt=capi.FILTER_EXACT)
    sub = subsystem_for_scene(s, luts=None, noise=oracle_noise)
    L = torch.zeros((54, 96, 4), device="cuda:0")
    T = torch.zeros_like(L)
    depth = torch.from_numpy(np.asarray(s.depth).reshape(54, 96)).to("cuda:0")
    view = capi.View(96, 54, depth.data_ptr(), L.data_ptr(), T.data_ptr(), None)

    def render(stream=None):
        call("psc_render", sub.handle, C.byref(view), 1, C.c_void_p(stream.cuda_stream if stream else None))

    try:
        render()
        torch.cuda.synchronize()
        want = L.cpu().numpy(), T.cpu().numpy()
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            render(stream)
        o = capi.MarchOptions.from_buffer_copy(sub.options)
        o.storage = then
        sub.set_options(o)
        render()
        torch.cuda.synchronize()
        L.zero_()
        T.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert want[0].any()
        assert np.array_equal(L.cpu().numpy(), want[0]) and np.array_equal(T.cpu().numpy(), want[1])
        del graph
    finally:
        sub.close()
