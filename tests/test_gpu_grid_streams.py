"""Grid calls of one context on two streams share its staged corner quads: each
call waits for the one before it.  Two grids of different density, their layer
gradients queued in turn on two streams without a synchronisation between
them, against each grid alone.  The sums' order changes their last bits (1e-12
of their terms, which cancel to about 1e-3); a mixed-up grid is off by its
density's factor of three: 1e-6."""
import numpy as np
import pytest

from pedalsky_b200 import grid as GR

from .test_gpu_grid_edges import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(33, 9, 2), (64, 8, 65)])
def test_two_streams(oracle, oracle_noise, shape):
    torch, sc, luts, G, spec, sub, P, tgt = _problem(oracle, oracle_noise, shape, 40, 6, 35.0, 0.5)
    try:
        Q = GR.GridProblem(sc, G * np.float32(3.0), spec=spec)
        Q.set_target(tgt)
        alone = []
        for R in (P, Q):
            out = torch.zeros(2, dtype=torch.float64, device="cuda:0")
            R.layer_gradient(sub.handle, out)
            torch.cuda.synchronize()
            alone.append(out.cpu().numpy())
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        outs = [torch.zeros((8, 2), dtype=torch.float64, device="cuda:0") for _ in streams]
        torch.cuda.synchronize()
        for i in range(8):
            for R, s, o in zip((P, Q), streams, outs):
                R.layer_gradient(sub.handle, o[i], stream=s)
        torch.cuda.synchronize()
    finally:
        sub.close()
    for o, a in zip(outs, alone):
        assert np.linalg.norm(a) > 0
        np.testing.assert_allclose(o.cpu().numpy(), np.tile(a, (8, 1)), rtol=1e-6, atol=1e-6 * np.abs(a).max())
