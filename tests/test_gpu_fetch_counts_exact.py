"""psc_count_fetches with exact filtering counts the light taps that are
fetched: those whose profile exceeds 1 - coverage, along the straight light path
and in the cone, against the FP64 oracle's count.  The dense samples agree to
1e-3 and FP32 heights move a few taps across the profile's border: 2e-3."""
import pytest

from pedalsky_b200 import capi, scenes

from .test_gpu_fetch_counts import _render_and_count

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["u8", "f16"])
@pytest.mark.parametrize("cone", [0, 1])
def test_light_taps_match_the_oracle(oracle, oracle_noise, storage, cone):
    s = scenes.precision_1080p(160, 90, storage=capi.STORAGE_NAMES[storage], schedule=capi.SCHED_FAST,
                               filt=capi.FILTER_NAMES["exact"])
    s.params.cone_light_sampling = cone
    _, _, c = _render_and_count(s, count=True)
    luts = oracle.bake_luts(s.frame, s.world)
    _, _, oc = oracle.render(s, oracle_noise, luts, precision=oracle.FP64, counters=True)
    print(storage, cone, c["light_taps"], oc["light_live"], oc["light"])
    assert abs(c["dense_samples"] - oc["dense"]) <= 1e-3 * oc["dense"]
    assert oc["light_live"] < 0.95 * oc["light"]
    assert abs(c["light_taps"] - oc["light_live"]) <= 2e-3 * oc["light_live"]
