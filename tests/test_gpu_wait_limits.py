"""The bounded waits inside the circuits' kernels run out (a limit of no
polls): the kernels wait for their copies and return, the call ends with
FQ_ERR_TIMEOUT, and the next circuits of the context, replays of captured
ones among them, give what they gave before."""
import numpy as np
import pytest

from conftest import angles, assert_state_close, complete_int

pytestmark = pytest.mark.gpu


# 16, 19: a grid barrier (64 CTAs, 128 CTAs of another tile size); 24, 26: TMA
# pipelines, of warps and of CTAs.
@pytest.mark.parametrize("n", [16, 19, 24, 26])
def test_waits_give_up_and_later_circuits_are_right(fq, oracle, n):
    import torch
    rng = np.random.default_rng(n)
    W, (g, b) = complete_int(n, rng), angles(rng, 3)
    lib = fq.lib()
    stream = torch.cuda.Stream()
    with fq.Context(0, stream.cuda_stream) as c:
        st = c.state(n)
        try:
            e = c.qaoa_forward(st, W, g, b)
            want_e = st.to_host()
            c.qaoa_forward(st, W, g, b, energy=False)  # another last pass, other roundings
            want = st.to_host()
            if n < 20:
                assert_state_close(want, oracle.qaoa_logical(W, g, b), what=f"N={n}")
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                c.qaoa_forward(st, W, g, b, energy=False)
            for energy in (True, False):
                assert lib.fq_ctx_selftest_polls(c.handle, 0) == fq.OK
                with pytest.raises(fq.FQError) as err:
                    c.qaoa_forward(st, W, g, b, energy=energy)
                    c.synchronize()
                assert err.value.status == fq.ERR_TIMEOUT
                assert lib.fq_ctx_selftest_polls(c.handle, -1) == fq.OK
                graph.replay()
                torch.cuda.synchronize()
                assert np.array_equal(st.to_host(), want)
                assert c.qaoa_forward(st, W, g, b) == e
                assert np.array_equal(st.to_host(), want_e)
        finally:
            st.free()
