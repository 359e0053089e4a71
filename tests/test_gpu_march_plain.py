"""GPU tests of the PLAIN march's branches that the other tests leave out:
octaves past the ones whose phase values are kept per layer (8), with a
Cumulonimbus layer whose droplet size changes with height (values below, inside
and above the blend band), weather maps that are not uniform (square and not a
power of two), and an extinction so strong that the profile bound lies close to
the density threshold.  Against the FP64 oracle at the parity bar of the other
march tests: p99.9 within 1e-3, mean within 1e-4."""
import numpy as np
import pytest

from pedalsky_b200 import capi, scenes

from . import _gpu
from ._metrics import composite, rel_stats

pytestmark = pytest.mark.gpu

CB = [(0, 1500.0, 2300.0, 0.5), (7, 3000.0, 11000.0, 0.7)]


def _weather(s, w, h):
    rng = np.random.default_rng(w * 1000 + h)
    s.weather, s.weather_w, s.weather_h = rng.uniform(0.0, 1.0, (h, w)).astype(np.float32).reshape(-1), w, h
    s.weather_format = capi.WEATHER_R32F


def _thin(s):
    for i in range(s.n_layers):
        s.layers[i].density_scale = 0.004  # the 1e-3 threshold is a quarter of it


@pytest.mark.parametrize("storage", ["u8", "f32"])
@pytest.mark.parametrize("case,layers,octaves,change", [
    ("ten_octaves", CB, 10, lambda s: None),
    ("one_octave", CB, 1, lambda s: None),
    ("weather_100x60", CB, 4, lambda s: _weather(s, 100, 60)),
    ("weather_1x1", CB[:1], 3, lambda s: _weather(s, 1, 1)),
    ("thin", CB[:1], 4, _thin),
])
def test_plain_branches_match_fp64(oracle, oracle_noise, case, layers, octaves, change, storage):
    s = scenes.precision_1080p(96, 54, storage=capi.STORAGE_NAMES[storage], schedule=capi.SCHED_PLAIN)
    s.layers, s.n_layers = scenes.synth_layers(layers)
    s.params.cloud_layer_count = s.n_layers
    s.params.multi_scatter_octaves = octaves
    change(s)
    luts = oracle.bake_luts(s.frame, s.world)
    L, T = oracle.render(s, oracle_noise, luts)
    _, _, hdr = _gpu.render(s, oracle_noise, luts, composite_bg=s.background)
    st = rel_stats(hdr, composite(L, T, s.background))
    print(case, storage, st)
    assert np.isfinite(hdr).all()
    assert st["p999"] <= 1e-3 and st["mean"] <= 1e-4, st
