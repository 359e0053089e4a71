"""GPU tests of the voxel-grid kernels where their padded layout and their
skipping of empty samples can go wrong: grids of one cell, of odd and thin
shapes, views whose rays pass beside the grid, low sun (light paths past
20 km, and a sun below the horizon), step and light-step counts that leave
remainders in the groups the kernels fetch, and grids that hold an infinity.

Forward image and gradient against the FP64 oracle.  Tolerances: FP32
positions on paths of up to 30 km resolve 2e-3 m and the smallest cells here
are 60 m wide, so a trilinear weight is off by up to 3e-5 and a grid value by
that share of its neighbours' difference; the sums over a ray average that
down, and the bars are 1e-3 of the image (L2) and 4e-3 of the gradient (L2),
as the full-size test's 2e-3 for cells of 78 m and paths of 5 km."""
import numpy as np
import pytest

from pedalsky_b200 import grid as GR
from pedalsky_b200 import scenes
from pedalsky_b200.subsystem import subsystem_for_scene

from . import _gpu
from ._metrics import composite

pytestmark = pytest.mark.gpu

W, H = 40, 24


def _problem(oracle, oracle_noise, shape, steps, light, sun_alt, fill):
    torch = _gpu.torch_cuda()
    sc = scenes.grid_512(W, H, grid_shape=(4, 4, 4), steps=steps)
    sc.params.light_steps = light
    sc.frame = scenes.frame_for(W, H, pitch_deg=55.0, fov_deg=60.0, sun_alt_deg=sun_alt)
    luts = oracle.bake_luts(sc.frame, sc.world)
    nx, ny, nz = shape
    rng = np.random.default_rng(nx * 1000 + ny * 100 + nz)
    G = (rng.uniform(0.0, 0.004, (ny, nz, nx)) * (rng.uniform(size=(ny, nz, nx)) < fill)).astype(np.float32)
    spec = dict(sc.extra["grid_spec"], exit_transmittance=0.0)
    sub = subsystem_for_scene(sc, luts=luts, noise=oracle_noise)
    P = GR.GridProblem(sc, G, spec=spec)
    tgt = (np.asarray(sc.background) * np.float32(0.7)).astype(np.float32)
    P.set_target(tgt)
    return torch, sc, luts, G, spec, sub, P, tgt


@pytest.mark.parametrize("shape,steps,light,sun_alt,fill", [
    ((1, 1, 1), 17, 6, 35.0, 1.0),
    ((5, 3, 7), 96, 1, 35.0, 0.6),
    ((33, 9, 2), 61, 4, 60.0, 0.3),
    ((2, 31, 33), 8, 7, 3.0, 0.3),
    ((64, 1, 65), 97, 6, 1.0, 0.2),
    ((31, 16, 17), 40, 5, -4.0, 0.3),
])
def test_edges_match_fp64(oracle, oracle_noise, shape, steps, light, sun_alt, fill):
    torch, sc, luts, G, spec, sub, P, tgt = _problem(oracle, oracle_noise, shape, steps, light, sun_alt, fill)
    try:
        P.render(sub.handle)
        torch.cuda.synchronize()
        img = composite(P.L.cpu().numpy(), P.T.cpu().numpy(), sc.background)[..., :3]
        P.zero_grad()
        P.adjoint(sub.handle)
        torch.cuda.synchronize()
        g, acc = P.grad.cpu().numpy().astype(np.float64), P.acc.cpu().numpy()
    finally:
        sub.close()
    Lo, To = oracle.grid_render(sc, oracle_noise, luts, G, spec)
    ref = composite(Lo, To, sc.background)[..., :3]
    e = np.linalg.norm(img - ref) / np.linalg.norm(ref)
    go, gso, lo = oracle.grid_adjoint(sc, oracle_noise, luts, G, spec, sc.background, tgt, threads=4)
    eg = np.linalg.norm(g - go) / np.linalg.norm(go)
    print(f"{shape}: image {e:.2e}, gradient {eg:.2e}, loss {acc[0]} vs {lo}, scale {acc[1]} vs {gso}")
    assert e <= 1e-3, e
    assert eg <= 4e-3, eg
    assert abs(acc[0] - lo) <= 2e-3 * lo
    assert abs(acc[1] - gso) <= 1e-2 * abs(gso)


def test_infinite_cell_keeps_every_sample_lit(oracle, oracle_noise):
    """An infinity reaches the image through the light sum of empty samples
    too: a grid that is empty but for one infinite cell gives no finite pixel
    where the cell shades or lies on the ray, and the empty grid's image
    elsewhere."""
    torch, sc, luts, G, spec, sub, P, _ = _problem(oracle, oracle_noise, (9, 5, 9), 40, 6, 35.0, 0.0)
    try:
        P.render(sub.handle)
        clear = P.L.cpu().numpy()
        P.values[2, 4, 4] = float("inf")
        P.render(sub.handle)
        torch.cuda.synchronize()
        L = P.L.cpu().numpy()[..., :3]
    finally:
        sub.close()
    assert not clear[..., :3].any()
    bad = ~np.isfinite(L).all(-1)
    assert bad.any()
    assert not L[~bad].any()


def test_wide_grid_matches_narrow_grid(oracle, oracle_noise):
    """A row of 2^21 cells takes the kernels that count cells without the
    mantissa trick; of constant value it is the same cloud as a row of 8 cells
    over the view (both are constant there), so images, losses and the summed
    gradients agree to FP32 rounding over about 40 samples: 1e-4."""
    torch = _gpu.torch_cuda()
    sc = scenes.grid_512(W, H, grid_shape=(4, 4, 4), steps=16)
    sc.frame = scenes.frame_for(W, H, pitch_deg=65.0, fov_deg=40.0, sun_alt_deg=70.0)
    luts = oracle.bake_luts(sc.frame, sc.world)
    sub = subsystem_for_scene(sc, luts=luts, noise=oracle_noise)
    got = []
    try:
        for nx in (8, 1 << 21):
            P = GR.GridProblem(sc, np.full((1, 8, nx), 5e-4, np.float32))
            P.set_target((np.asarray(sc.background) * np.float32(0.7)).astype(np.float32))
            P.render(sub.handle)
            img = P.composite_image().cpu().numpy()[..., :3]
            P.zero_grad()
            P.adjoint(sub.handle)
            torch.cuda.synchronize()
            got.append((img, float(P.grad.double().sum()), P.acc.cpu().numpy()))
            del P
    finally:
        sub.close()
    (a, ga, aa), (b, gb, ab) = got
    assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(a)
    assert abs(ga - gb) <= 1e-4 * abs(ga)
    np.testing.assert_allclose(ab, aa, rtol=1e-4)


@pytest.mark.parametrize("shape,steps,light", [((5, 3, 7), 23, 6), ((33, 9, 2), 40, 5), ((64, 1, 65), 17, 1)])
def test_range_gradient_of_an_embedded_grid(oracle, oracle_noise, shape, steps, light):
    """A ring of empty cells around a grid (its extent grown by as much) is
    the same cloud, so the gradient in the layer's base and top is the same.
    The grid's slopes jump at cell borders and the two sets of cell
    coordinates round apart by about 1e-5 cells: of the 3e5 taps of this view
    a few change cells, each worth at most 1e-3 of the sum: 1e-2."""
    torch, sc, luts, G, spec, sub, P, tgt = _problem(oracle, oracle_noise, shape, steps, light, 35.0, 0.5)
    ring = np.pad(G, ((0, 0), (1, 1), (1, 1)))
    cx, cz = spec["size_x_m"] / shape[0], spec["size_z_m"] / shape[2]
    grown = dict(spec, min_x_m=spec["min_x_m"] - cx, min_z_m=spec["min_z_m"] - cz, size_x_m=spec["size_x_m"] + 2 * cx,
                 size_z_m=spec["size_z_m"] + 2 * cz)
    got = []
    try:
        for Q in (P, GR.GridProblem(sc, ring, spec=grown)):
            Q.set_target(tgt)
            out = torch.zeros(2, dtype=torch.float64, device="cuda:0")
            Q.layer_gradient(sub.handle, out)
            torch.cuda.synchronize()
            got.append(out.cpu().numpy())
    finally:
        sub.close()
    print(shape, got)
    assert np.abs(got[0]).min() > 0
    assert np.linalg.norm(got[0] - got[1]) <= 1e-2 * np.linalg.norm(got[0])
