"""Cone light sampling of the FAST schedule under Cumulonimbus layers, whose
taps are taken without a look at the profile first, and beside a layer of another type, whose
are not: against the FP64 oracle at the parity bar of the other march tests,
p99.9 within 1e-3 and mean within 1e-4."""
import numpy as np
import pytest

from pedalsky_b200 import capi, scenes

from . import _gpu
from ._metrics import composite, rel_stats

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["u8", "f32"])
@pytest.mark.parametrize("layers", [[(7, 900.0, 9000.0, 0.7)], [(0, 1500.0, 2300.0, 0.5), (7, 3000.0, 11000.0, 0.4)]])
def test_cone_under_cumulonimbus_matches_fp64(oracle, oracle_noise, layers, storage):
    s = scenes.precision_1080p(96, 54, storage=capi.STORAGE_NAMES[storage], schedule=capi.SCHED_FAST,
                               filt=capi.FILTER_EXACT)
    s.layers, s.n_layers = scenes.synth_layers(layers)
    s.params.cloud_layer_count = s.n_layers
    s.params.cone_light_sampling = 1
    luts = oracle.bake_luts(s.frame, s.world)
    L, T = oracle.render(s, oracle_noise, luts)
    _, _, hdr = _gpu.render(s, oracle_noise, luts, composite_bg=s.background)
    st = rel_stats(hdr, composite(L, T, s.background))
    print(len(layers), storage, st)
    assert np.isfinite(hdr).all()
    assert st["p999"] <= 1e-3 and st["mean"] <= 1e-4, st
