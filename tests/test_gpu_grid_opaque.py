"""The adjoint of a grid that holds cells more opaque by many powers of ten than
the rest: the transmittance before a step is taken from a running sum of the
grid values, and the values in front of an opaque cell must not be lost in it.

Against the FP64 oracle at 2e-2 of the gradient (L2): FP32 positions put a
sample on the other side of an opaque cell's border (its weight times 1e16 is
opaque wherever it is not 0) for about 3e-5 of the samples, one or two rays of
the hundreds that meet the cell, each worth about 1 % of the cells it crosses."""
import numpy as np
import pytest

from pedalsky_b200 import grid as GR

from .test_gpu_grid_edges import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opaque", [1e3, 1e16])
def test_gradient_in_front_of_an_opaque_cell(oracle, oracle_noise, opaque):
    torch, sc, luts, G, spec, sub, _, tgt = _problem(oracle, oracle_noise, (6, 5, 6), 48, 4, 45.0, 1.0)
    G = G * np.float32(0.2)
    G[2:4, 2:4, 2:4] = opaque
    try:
        P = GR.GridProblem(sc, G, spec=spec)
        P.set_target(tgt)
        P.adjoint(sub.handle)
        torch.cuda.synchronize()
        g = P.grad.cpu().numpy().astype(np.float64)
    finally:
        sub.close()
    go, _, _ = oracle.grid_adjoint(sc, oracle_noise, luts, G, spec, sc.background, tgt, threads=4)
    assert np.isfinite(go).all() and np.isfinite(g).all()
    thin = G < opaque
    e = np.linalg.norm((g - go)[thin]) / np.linalg.norm(go[thin])
    print(f"opaque {opaque:g}: {e:.2e}")
    assert e <= 2e-2, e
