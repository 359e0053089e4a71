"""The FAST march of Cumulonimbus scenes takes another form for launches of at
most 1036 CTAs (16x8 pixels each, 7 per SM): a frame of 1089 CTAs against its
bands of one row of CTAs (33), of the most that still take that form (1023) and of the first
that does not (1056).  A frame split into bands is the frame rendered whole, bit for bit,
so the forms' images have to be equal."""
import ctypes as C

import numpy as np
import pytest

from pedalsky_b200 import capi, scenes
from pedalsky_b200.capi import call
from pedalsky_b200.subsystem import subsystem_for_scene

from . import _gpu

pytestmark = pytest.mark.gpu

W, H = 33 * 16, 33 * 8


@pytest.mark.parametrize("storage,filt", [(capi.STORAGE_F16, capi.FILTER_HYBRID), (capi.STORAGE_U8, capi.FILTER_EXACT),
                                          (capi.STORAGE_BF16, capi.FILTER_EXACT)])
def test_bands_match_the_frame(oracle_noise, storage, filt):
    torch = _gpu.torch_cuda()
    s = scenes.stress_2160p(W, H, frame_index=0, schedule=capi.SCHED_FAST, storage=storage, filt=filt)
    sub = subsystem_for_scene(s, luts=None, noise=oracle_noise)
    depth = torch.from_numpy(np.asarray(s.depth).reshape(H, W)).to("cuda:0")

    def band(y0, rows):
        d = depth[y0:y0 + rows].contiguous()
        L = torch.zeros((rows, W, 4), device="cuda:0")
        T = torch.zeros((rows, W, 4), device="cuda:0")
        v = capi.View(W, rows, d.data_ptr(), L.data_ptr(), T.data_ptr(), None, W, H, 0, y0)
        torch.cuda.synchronize()
        call("psc_render", sub.handle, C.byref(v), 1, None)
        torch.cuda.synchronize()
        return np.concatenate([L.cpu().numpy(), T.cpu().numpy()], axis=-1)

    try:
        whole = band(0, H)
        assert whole[..., 0].max() > 0 and whole[..., 4].min() < 0.5
        for y0, rows in ((40, 8), (0, 31 * 8), (16, 31 * 8), (8, 32 * 8)):
            assert np.array_equal(band(y0, rows), whole[y0:y0 + rows]), (y0, rows)
    finally:
        sub.close()
