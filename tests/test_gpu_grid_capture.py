"""Captured grid calls have scratch of their own: a graph replays into memory
that no other call of the context uses, and that stays while the graph does.
Against the same calls queued on their own.  The images are equal to the bit;
the gradients' sums change their last bits with their order (1e-12 of their
terms in FP64, 1e-6 in the FP32 grid gradient), where another grid's values
would show as its density's factor of three."""
import numpy as np
import pytest

from pedalsky_b200 import grid as GR

from .test_gpu_grid_edges import _problem

pytestmark = pytest.mark.gpu


def _capture(torch, stream, work):
    g = torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=stream):
        work(stream)
    return g


def _setup(oracle, oracle_noise, shape):
    torch, sc, luts, G, spec, sub, P, tgt = _problem(oracle, oracle_noise, shape, 40, 6, 35.0, 0.5)
    Q = GR.GridProblem(sc, G * np.float32(3.0), spec=spec)
    big = GR.GridProblem(sc, np.full((40, 90, 91), 1e-4, np.float32), spec=spec)
    for R in (Q, big):
        R.set_target(tgt)
    return torch, sub, P, Q, big


def _range(torch, R, sub, out, stream=None):
    R.layer_gradient(sub.handle, out, stream=stream)


def _alone(torch, sub, problems):
    want = []
    for R in problems:
        out = torch.zeros(2, dtype=torch.float64, device="cuda:0")
        _range(torch, R, sub, out)
        R.zero_grad()
        R.adjoint(sub.handle)
        R.render(sub.handle)
        torch.cuda.synchronize()
        want.append((out.cpu().numpy(), R.grad.cpu().numpy(), R.acc.cpu().numpy(), R.L.cpu().numpy()))
    return want


def _same(torch, R, out, want, times):
    torch.cuda.synchronize()
    o, g, acc, L = want
    np.testing.assert_allclose(out.cpu().numpy(), times * o, rtol=1e-6, atol=1e-6 * np.abs(times * o).max())
    np.testing.assert_allclose(R.grad.cpu().numpy(), times * g, rtol=1e-4, atol=1e-5 * np.abs(times * g).max())
    np.testing.assert_allclose(R.acc.cpu().numpy(), times * acc, rtol=1e-6)
    assert np.array_equal(R.L.cpu().numpy(), L)


@pytest.mark.parametrize("shape", [(33, 9, 2), (64, 8, 65)])
def test_graphs_beside_each_other_and_beside_larger_grids(oracle, oracle_noise, shape):
    torch, sub, P, Q, big = _setup(oracle, oracle_noise, shape)
    try:
        want = _alone(torch, sub, (P, Q))
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        outs = [torch.zeros(2, dtype=torch.float64, device="cuda:0") for _ in streams]
        torch.cuda.synchronize()
        graphs = []
        for R, s, o in zip((P, Q), streams, outs):
            def work(stream, R=R, o=o):
                _range(torch, R, sub, o, stream)
                R.adjoint(sub.handle, stream=stream)
                R.render(sub.handle, stream=stream)
            graphs.append(_capture(torch, s, work))
        for R in (P, Q):
            R.zero_grad()
        big.zero_grad()
        torch.cuda.synchronize()
        for _ in range(4):
            for g, s in zip(graphs, streams):
                with torch.cuda.stream(s):
                    g.replay()
            big.adjoint(sub.handle)  # grows the context's own scratch meanwhile
        for R, o, w in zip((P, Q), outs, want):
            _same(torch, R, o, w, 4)
        del graphs
    finally:
        sub.close()


def test_parallel_branches_of_one_capture(oracle, oracle_noise):
    torch, sub, P, Q, big = _setup(oracle, oracle_noise, (31, 16, 17))
    try:
        want = _alone(torch, sub, (P, Q))
        outs = [torch.zeros(2, dtype=torch.float64, device="cuda:0") for _ in range(2)]
        s, side = torch.cuda.Stream(), torch.cuda.Stream()
        for R in (P, Q):
            R.zero_grad()
        torch.cuda.synchronize()

        def work(stream):
            side.wait_stream(stream)
            for R, o, t in ((P, outs[0], stream), (Q, outs[1], side)):
                _range(torch, R, sub, o, t)
                R.adjoint(sub.handle, stream=t)
                R.render(sub.handle, stream=t)
            stream.wait_stream(side)
        g = _capture(torch, s, work)
        for _ in range(3):
            with torch.cuda.stream(s):
                g.replay()
        for R, o, w in zip((P, Q), outs, want):
            _same(torch, R, o, w, 3)
        del g
    finally:
        sub.close()


def test_scratch_of_destroyed_graphs_is_used_again(oracle, oracle_noise):
    """Thirty captures of a grid whose adjoint scratch is 1.3 GB, each graph
    destroyed before the next, hold three of them at most."""
    torch, sc, luts, G, spec, sub, P, tgt = _problem(oracle, oracle_noise, (4, 4, 4), 8, 2, 35.0, 0.5)
    try:
        R = GR.GridProblem(sc, np.full((64, 780, 780), 1e-5, np.float32), spec=spec)
        R.set_target(tgt)
        torch.cuda.synchronize()
        s = torch.cuda.Stream()
        free = []
        for _ in range(30):
            g = _capture(torch, s, lambda stream: R.adjoint(sub.handle, stream=stream))
            with torch.cuda.stream(s):
                g.replay()
            torch.cuda.synchronize()
            del g
            free.append(torch.cuda.mem_get_info()[0])
        assert free[0] - min(free) <= 3 * 1.4e9
        P.render(sub.handle)  # gives the idle scratch back
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] >= free[0]
    finally:
        sub.close()
