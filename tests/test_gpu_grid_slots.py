"""Grid calls in flight on several streams at once: more streams than the
context keeps scratch for, grids of different size and density, so that scratch
grows, is taken in turn and is waited for.  Every call against the same call
alone: images to the bit, gradients to their sums' order (1e-6; a mixed-up grid
is off by its density's factor)."""
import numpy as np
import pytest

from pedalsky_b200 import grid as GR

from .test_gpu_grid_edges import _problem

pytestmark = pytest.mark.gpu


def test_more_streams_than_slots(oracle, oracle_noise):
    torch, sc, luts, G, spec, sub, _, tgt = _problem(oracle, oracle_noise, (31, 16, 17), 40, 6, 35.0, 0.5)
    try:
        problems = []
        for i in range(11):
            R = GR.GridProblem(sc, np.repeat(G, 1 + i % 3, axis=1) * np.float32(1.0 + i), spec=spec)
            R.set_target(tgt)
            problems.append(R)
        want = []
        for R in problems:
            out = torch.zeros(2, dtype=torch.float64, device="cuda:0")
            R.layer_gradient(sub.handle, out)
            R.render(sub.handle)
            torch.cuda.synchronize()
            want.append((out.cpu().numpy(), R.L.cpu().numpy().copy()))
            R.L.zero_()
        streams = [torch.cuda.Stream() for _ in problems]
        outs = [torch.zeros((6, 2), dtype=torch.float64, device="cuda:0") for _ in problems]
        torch.cuda.synchronize()
        for i in range(6):
            for R, s, o in zip(problems, streams, outs):
                R.layer_gradient(sub.handle, o[i], stream=s)
                if i % 2:
                    R.render(sub.handle, stream=s)
        torch.cuda.synchronize()
    finally:
        sub.close()
    for R, o, (a, L) in zip(problems, outs, want):
        assert np.linalg.norm(a) > 0 and L.any()
        np.testing.assert_allclose(o.cpu().numpy(), np.tile(a, (6, 1)), rtol=1e-6, atol=1e-6 * np.abs(a).max())
        assert np.array_equal(R.L.cpu().numpy(), L)
