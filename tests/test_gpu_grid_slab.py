"""A large grid one cell high takes the kernels whose arrays hold only the
corners that exist: no more than 16 bytes of quads a cell (and its border) and
as much for the gradient, where two layers of zeros around it would take five
times that.  Image and gradient against the FP64 oracle; the cells are 7 m wide,
FP32 positions on these paths resolve 2e-3 m, so a trilinear weight is off by
3e-4 and, the values changing over 400 m, a grid value by 1e-5: 1e-3 of the image (L2),
4e-3 of the gradient (L2)."""
import numpy as np
import pytest

from pedalsky_b200 import grid as GR

from ._metrics import composite
from .test_gpu_grid_edges import _problem

pytestmark = pytest.mark.gpu

N = 2900


def test_slab_memory_and_gradient(oracle, oracle_noise):
    torch, sc, luts, _, spec, sub, _, tgt = _problem(oracle, oracle_noise, (4, 4, 4), 48, 5, 40.0, 0.5)
    a = np.sin(np.arange(N) * (2 * np.pi / 58)).astype(np.float32)
    G = (0.001 + 0.0008 * a[None, :, None] * a[None, None, :]).astype(np.float32)
    try:
        P = GR.GridProblem(sc, G, spec=spec)
        P.set_target(tgt)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        P.render(sub.handle)
        P.adjoint(sub.handle)
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info()[0]
        img = composite(P.L.cpu().numpy(), P.T.cpu().numpy(), sc.background)[..., :3]
        g = P.grad.cpu().numpy().astype(np.float64)
    finally:
        sub.close()
    Lo, To = oracle.grid_render(sc, oracle_noise, luts, G, spec)
    ref = composite(Lo, To, sc.background)[..., :3]
    go, _, _ = oracle.grid_adjoint(sc, oracle_noise, luts, G, spec, sc.background, tgt, threads=1)
    e = np.linalg.norm(img - ref) / np.linalg.norm(ref)
    eg = np.linalg.norm(g - go) / np.linalg.norm(go)
    print(f"image {e:.2e}, gradient {eg:.2e}, scratch {used / 1e6:.0f} MB")
    assert e <= 1e-3 and eg <= 4e-3
    assert used <= 2 * 16 * (N + 1) ** 2 + 64e6
