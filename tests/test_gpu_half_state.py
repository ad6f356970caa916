"""GPU parity of whole circuits and gradients on half states: only the
amplitudes with qubit N-1 = 0 are swept.  N = 16..19 as one cooperative
launch (every CTA size, even and odd P), N >= 20 as passes at the edges of
their tile geometries: rows of 16 amplitudes (N=20), paired rows of 8 and 4
(N=21, 22), the first size with three passes per layer (N=23), the mirror
pass as the last pass, and more layers than either keeps tables for."""
import numpy as np
import pytest

from conftest import (ENERGY_RTOL, GRAD_TOL, angles, assert_state_close, complete_int, gnp_fp,
                      gnp_int)

pytestmark = pytest.mark.gpu

WIDE = 300000  # |w| up to this: integer weights beyond every phase table


def graph(kind, n, rng):
    if kind == "fp":
        return gnp_fp(n, rng)
    if kind == "wide":
        return gnp_int(n, rng, lo=-WIDE, hi=WIDE)
    return complete_int(n, rng, -7, 9)


@pytest.mark.parametrize("n,P,kind", [(16, 3, "int"), (16, 2, "wide"), (17, 1, "int"),
                                      (17, 2, "fp"), (17, 7, "int"), (18, 1, "fp"),
                                      (18, 2, "wide"), (19, 3, "int"), (20, 1, "fp"),
                                      (21, 2, "int"), (22, 1, "int"), (22, 2, "fp"),
                                      (23, 1, "fp"), (23, 2, "int"),
                                      # more layers than the shared layer tables hold
                                      (17, 66, "fp"), (17, 65, "int"), (17, 40, "int")])
def test_half_state_forward(ctx, oracle, n, P, kind):
    rng = np.random.default_rng(1000 * n + P)
    W = graph(kind, n, rng)
    g, b = angles(rng, P)
    if kind == "wide":
        g /= WIDE  # keep gamma * W at ordinary size
    st = ctx.state(n)
    try:
        e = ctx.qaoa_forward(st, W, g, b)
        psi = st.to_host()
    finally:
        st.free()
    want = oracle.qaoa_logical(W, g, b)
    assert_state_close(psi, want, what=f"N={n} P={P} {kind}")
    eo = oracle.expectation(want, W)
    assert abs(e - eo) <= ENERGY_RTOL * max(1.0, abs(eo), np.abs(W).sum())


@pytest.mark.parametrize("n,P,kind", [(16, 4, "fp"), (17, 1, "fp"), (18, 2, "int"),
                                      (17, 3, "wide"), (19, 3, "int"), (17, 36, "int"),
                                      (17, 65, "fp"),
                                      (20, 1, "int"), (21, 2, "fp")])
def test_half_state_gradient(ctx, oracle, n, P, kind):
    rng = np.random.default_rng(2000 * n + P)
    W = graph(kind, n, rng)
    g, b = angles(rng, P)
    if kind == "wide":
        g /= WIDE
    e, gg, gb = ctx.energy_grad(n, W, g, b)
    eo, go, bo = oracle.energy_grad(W, g, b)
    scale = max(1.0, np.abs(go).max(), np.abs(bo).max())
    assert abs(e - eo) <= ENERGY_RTOL * max(1.0, abs(eo), np.abs(W).sum())
    assert np.abs(gg - go).max() <= GRAD_TOL * scale
    assert np.abs(gb - bo).max() <= GRAD_TOL * scale


@pytest.mark.parametrize("n", [12, 14, 17, 18])
def test_captured_circuit_replays(fq, oracle, n):
    """A circuit captured in a CUDA graph gives the same state at every
    replay (the grid barrier of one launch leaves itself ready for the next)."""
    import torch
    rng = np.random.default_rng(n)
    W = complete_int(n, rng)
    g, b = angles(rng, 3)
    want = oracle.qaoa_logical(W, g, b)
    stream = torch.cuda.Stream()
    with fq.Context(0, stream.cuda_stream) as c:
        st = c.state(n)
        try:
            c.qaoa_forward(st, W, g, b)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                c.qaoa_forward(st, W, g, b, energy=False)
            for _ in range(3):
                st.init_basis0()
                c.synchronize()
                graph.replay()
                torch.cuda.synchronize()
                assert_state_close(st.to_host(), want, what=f"N={n}")
        finally:
            st.free()
