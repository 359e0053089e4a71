"""The rule that picks the 8-bit kernels for texel coordinates past 2^22: times
either side of the line where a 10 m/s wind carries the detail noise over it
(1.05e7 s, less the planet's extent), and noise scales so small that the
planet's extent alone reaches it.  8-bit against FP32 volumes as in
test_gpu_march_far.py; a batch with views on both sides against its views
rendered alone; and a captured batch whose view crosses the line."""
import numpy as np
import pytest

from pedalsky_b200 import batch as B
from pedalsky_b200 import capi, scenes
from pedalsky_b200.subsystem import subsystem_for_scene

from . import _gpu
from ._metrics import rel_stats
from .test_gpu_batch import _compare, _run_batch
from .test_gpu_fetch_counts import _render_and_count

pytestmark = pytest.mark.gpu


def _drift(s, seconds):
    s.params.wind_drift_strength = 1.0
    s.frame.simulated_seconds = seconds
    s.wind = scenes.wind_field(10.0, 230.0)
    return s


@pytest.mark.parametrize("schedule", [capi.SCHED_PLAIN, capi.SCHED_FAST])
@pytest.mark.parametrize("seconds,base,detail", [(9.0e6, 4500.0, 800.0), (1.02e7, 4500.0, 800.0),
                                                 (1.2e7, 4500.0, 800.0), (0.0, 350.0, 90.0)])
def test_either_side_of_the_line(oracle, oracle_noise, schedule, seconds, base, detail):
    got = []
    for storage in (capi.STORAGE_U8, capi.STORAGE_F32):
        s = _drift(scenes.precision_1080p(96, 54, storage=storage, schedule=schedule, filt=capi.FILTER_EXACT), seconds)
        s.params.base_scale_m, s.params.detail_scale_m = base, detail
        luts = oracle.bake_luts(s.frame, s.world)
        _, T, hdr = _gpu.render(s, oracle_noise, luts, composite_bg=s.background)
        got.append(hdr)
        assert T[..., :3].min() < 0.9
    st = rel_stats(got[0], got[1])
    print(schedule, seconds, base, detail, st)
    assert st["p999"] <= 1e-3 and st["mean"] <= 1e-4, st


@pytest.fixture(scope="module")
def views():
    out = scenes.batch_views(4, seed=7, size_scale=0.06, storage=capi.STORAGE_U8, filt=capi.FILTER_EXACT)
    return [_drift(s, 5e7 if i == 2 else 1e5) for i, s in enumerate(out)]


@pytest.mark.parametrize("form", [capi.BATCH_PERSISTENT, capi.BATCH_PER_VIEW])
def test_batch_with_views_on_both_sides(views, oracle_noise, form):
    _compare(views, _run_batch(views, oracle_noise, (128, 16, 1, form), reps=2), oracle_noise)


@pytest.mark.parametrize("form", [capi.BATCH_PERSISTENT, capi.BATCH_PER_VIEW])
def test_captured_batch_follows_a_view_over_the_line(views, oracle_noise, form):
    torch = _gpu.torch_cuda()
    near, far = views[:2], _run_batch(views[2:3] + views[:1], oracle_noise)[0]
    sub = subsystem_for_scene(views[0], luts=None, noise=oracle_noise)
    try:
        b = B.Batch([views[2], views[0]], "cuda:0", outputs=("luminance", "transmittance"))
        B.set_tuning(sub.handle, 128, 16, 1, form)
        b.arr[0].frame.simulated_seconds = near[0].frame.simulated_seconds
        b.render(sub.handle)
        torch.cuda.synchronize()
        assert not np.array_equal(b.trans[0].cpu().numpy(), far[1])
        b.arr[0].frame.simulated_seconds = 5e7
        b.render(sub.handle)
        torch.cuda.synchronize()
        assert np.array_equal(b.trans[0].cpu().numpy(), far[1])
    finally:
        sub.close()


def test_counting_build_past_the_line():
    s = _drift(scenes.precision_1080p(160, 90, storage=capi.STORAGE_U8, schedule=capi.SCHED_FAST,
                                      filt=capi.FILTER_EXACT), 5e7)
    L0, T0, _ = _render_and_count(s, count=False)
    L1, T1, c = _render_and_count(s, count=True)
    # the instrumented build computes the same image
    assert np.abs(L1 - L0).max() <= 1e-6 * max(np.abs(L0).max(), 1.0)
    assert np.abs(T1 - T0).max() <= 1e-6 and c["light_taps"] > 0
