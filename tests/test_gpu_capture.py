"""Circuits captured in a CUDA graph as the first call of their context,
called as usual before the graph runs, and replayed in turn with calls:
always the oracle's state."""
import numpy as np
import pytest

from conftest import angles, assert_state_close, complete_int

pytestmark = pytest.mark.gpu


class Captured:
    def __init__(self, ctx, stream, st, W, g, b):
        import torch
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph, stream=stream):
            ctx.qaoa_forward(st, W, g, b, energy=False)

    def replay(self):
        import torch
        self.graph.replay()
        torch.cuda.synchronize()


def context(fq):
    import torch
    stream = torch.cuda.Stream()
    return stream, fq.Context(0, stream.cuda_stream)


@pytest.mark.parametrize("n", [16, 17, 19])
def test_capture_is_the_first_call(fq, oracle, n):
    rng = np.random.default_rng(n)
    W, (g, b) = complete_int(n, rng), angles(rng, 3)
    want = oracle.qaoa_logical(W, g, b)
    stream, ctx = context(fq)
    with ctx as c:
        st = c.state(n)
        try:
            cap = Captured(c, stream, st, W, g, b)
            for _ in range(2):
                c.qaoa_forward(st, W, g, b)
                assert_state_close(st.to_host(), want, what=f"N={n}, called")
                st.init_basis0()
                c.synchronize()
                cap.replay()
                assert_state_close(st.to_host(), want, what=f"N={n}, replayed")
        finally:
            st.free()


@pytest.mark.parametrize("n,P", [(9, 60), (12, 44), (14, 36), (15, 33), (3, 2100)])
def test_deep_small_circuits(fq, oracle, n, P):
    """More layers than the kernel parameters hold (and, last, than every
    context has room for): captured, replayed between calls of other circuits."""
    rng = np.random.default_rng(n)
    (W, V), (g, b) = (complete_int(n, rng) for _ in range(2)), angles(rng, P)
    want, other = oracle.qaoa_logical(W, g, b), oracle.qaoa_logical(V, b, g)
    stream, ctx = context(fq)
    with ctx as c:
        st = c.state(n)
        try:
            cap = Captured(c, stream, st, W, g, b)
            for _ in range(2):
                c.qaoa_forward(st, V, b, g)
                assert_state_close(st.to_host(), other, what=f"N={n}, called")
                cap.replay()
                assert_state_close(st.to_host(), want, what=f"N={n}, replayed")
        finally:
            st.free()


@pytest.mark.parametrize("n,P", [(16, 65), (20, 3), (21, 2)])
def test_replays_between_calls_on_other_graphs(fq, oracle, n, P):
    """Circuits as passes with tables (16 qubits: more layers than one launch
    holds): captured with only the weights in place, replayed between calls
    on another graph, and after the tables' buffer has been outgrown."""
    rng = np.random.default_rng(n + P)
    (W, V), (g, b) = (complete_int(n, rng) for _ in range(2)), angles(rng, P)
    want, other = oracle.qaoa_logical(W, g, b), oracle.qaoa_logical(V, g, b)
    big, (G, B) = complete_int(25, rng), angles(rng, 1)
    stream, ctx = context(fq)
    with ctx as c:
        st, st25 = c.state(n), c.state(25)
        try:
            st.init_basis0()
            c.expectation(st, W)  # the weights, nothing else
            cap = Captured(c, stream, st, W, g, b)
            c.qaoa_forward(st, W, g, b)
            assert_state_close(st.to_host(), want, what=f"N={n}, called first")
            for k in range(3):
                c.qaoa_forward(st, V, g, b)
                assert_state_close(st.to_host(), other, what=f"N={n}, called")
                if k == 1:
                    c.qaoa_forward(st25, big, G, B)
                cap.replay()
                assert_state_close(st.to_host(), want, what=f"N={n}, replayed")
        finally:
            st.free()
            st25.free()


def test_tables_grow_during_a_capture(fq):
    """The first call, captured, is of a size whose tables outgrow the
    context's: its replay gives the state of the call that follows."""
    n, P = 25, 2
    rng = np.random.default_rng(n)
    W, (g, b) = complete_int(n, rng), angles(rng, P)
    stream, ctx = context(fq)
    with ctx as c:
        st = c.state(n)
        try:
            cap = Captured(c, stream, st, W, g, b)
            c.qaoa_forward(st, W, g, b, energy=False)
            want = st.to_host()
            st.init_basis0()
            c.synchronize()
            cap.replay()
            assert np.array_equal(st.to_host(), want)
            assert abs(np.linalg.norm(want) - 1) <= 1e-12
        finally:
            st.free()
