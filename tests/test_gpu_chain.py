"""Passes launched in a chain (each may start while the one before it ends)
against the same passes launched one by one (a profiled context): the same
bits.  One tile per SM or less (N=20), up to two (N=21: the last size whose
adjoint passes chain), up to four (N=22: the last whose forward passes do),
more (N=23), and few tiles with more layers than one launch's tables hold
(N=17)."""
import numpy as np
import pytest

from conftest import angles, complete_int, gnp_fp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,P,kind", [(17, 66, "fp"), (20, 1, "int"), (20, 5, "int"),
                                      (20, 4, "fp"), (21, 2, "fp"), (21, 5, "int"),
                                      (22, 3, "int"), (23, 2, "fp")])
def test_chained_passes_match_single_launches(fq, n, P, kind):
    rng = np.random.default_rng(100 * n + P)
    # Graphs take turns, so that a table read too early would be another's.
    graphs = [gnp_fp(n, rng) if kind == "fp" else complete_int(n, rng, -7, 9) for _ in range(2)]
    sets = [angles(rng, P) for _ in range(2)]
    runs = []
    for one_by_one in (True, False):
        with fq.Context(0) as c:
            c.set_profiling(one_by_one)
            sv, cs = c.state(n), c.state(n)
            try:
                out = []
                for i in range(6):
                    W, (g, b) = graphs[i % 2], sets[i // 2 % 2]
                    e = c.qaoa_forward(sv, W, g, b)
                    psi = sv.to_host()
                    out.append((e, psi) + c.energy_grad(n, W, g, b, sv, cs))
            finally:
                sv.free()
                cs.free()
        runs.append(out)
    for a, b in zip(*runs):
        for x, y in zip(a, b):
            assert np.array_equal(np.asarray(x), np.asarray(y))


def test_threads_share_the_kernels(fq):
    """Contexts on threads of their own launch the same kernels with different
    amounts of shared memory (N=20: one CTA per SM) at the same time."""
    from concurrent.futures import ThreadPoolExecutor

    def work(n):
        rng = np.random.default_rng(n)
        W, (g, b) = complete_int(n, rng), angles(rng, 3)
        with fq.Context(0) as c:
            st = c.state(n)
            try:
                return {c.qaoa_forward(st, W, g, b) for _ in range(400)}
            finally:
                st.free()

    with ThreadPoolExecutor(4) as pool:
        res = list(pool.map(work, [20, 21, 20, 21]))
    assert all(len(r) == 1 for r in res)
    assert res[0] == res[2] and res[1] == res[3]


def test_captured_chain_replays(fq):
    """A chain captured in a CUDA graph gives the same state at each replay."""
    import torch
    n, rng = 20, np.random.default_rng(3)
    W, (g, b) = complete_int(n, rng), angles(rng, 4)
    stream = torch.cuda.Stream()
    with fq.Context(0, stream.cuda_stream) as c:
        st = c.state(n)
        try:
            c.qaoa_forward(st, W, g, b)
            want = st.to_host()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                c.qaoa_forward(st, W, g, b, energy=False)
            for _ in range(3):
                st.init_basis0()
                c.synchronize()
                graph.replay()
                torch.cuda.synchronize()
                assert np.array_equal(st.to_host(), want)
        finally:
            st.free()
