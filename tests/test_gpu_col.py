"""GPU parity of the fused pass of independent warps (k_pass_col: circuits of
24 and more qubits, rows of 8 to 128 amplitudes): every row width it takes,
both weight types, phases by product tree and per amplitude, against the
oracle where it is quick and against the reference schedule on the device."""
import numpy as np
import pytest

from conftest import ENERGY_RTOL, STATE_RTOL, angles, assert_state_close, complete_int, gnp_fp, gnp_int

pytestmark = pytest.mark.gpu

HUGE = 1 << 21  # integer-valued weights beyond the integer path: exact cut values in FP64


def graph(kind, n, rng):
    if kind == "fp":
        return gnp_fp(n, rng)
    if kind == "huge":
        return gnp_int(n, rng, lo=-HUGE, hi=HUGE)
    return complete_int(n, rng, -4, 10)


@pytest.mark.parametrize("P,kind", [(3, "int"), (2, "fp"), (2, "huge")])
def test_col_pass_against_oracle(ctx, oracle, P, kind):
    n = 24  # rows of 16 amplitudes, and of 256 on the general pass
    rng = np.random.default_rng(24 + P)
    W = graph(kind, n, rng)
    g, b = angles(rng, P)
    if kind == "huge":
        g *= 1e-5  # |gamma| sum|w| above the product-tree bound
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


@pytest.mark.parametrize("n,P,kind", [(25, 3, "int"), (26, 2, "fp"), (27, 3, "int"),
                                      (28, 2, "int"), (29, 2, "int"), (29, 3, "fp")])
def test_col_pass_against_reference_schedule(fq, ctx, n, P, kind):
    rng = np.random.default_rng(n)
    W = graph(kind, n, rng)
    g, b = angles(rng, P)
    C = 12
    a, r, x = ctx.state(n), ctx.state(n), ctx.state(n)
    try:
        ctx.qaoa_forward(a, W, g, b, energy=False)
        ctx.reference_schedule(r, W, C, g, b)
        ctx.permute_qubits(r, x, fq.reference_label_map(n, C, P))
        d = ctx.state_diff(a, x)
    finally:
        for s in (a, r, x):
            s.free()
    assert d["max_abs_diff"] <= STATE_RTOL * d["max_abs_b"]
    assert d["l2_diff"] <= STATE_RTOL * d["l2_b"]
