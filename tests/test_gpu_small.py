"""GPU parity of instances held on chip (one CTA up to 12 qubits, a
cluster of 2, 4 or 8 CTAs up to 15) at the edges of their layouts: states
smaller than the smallest CTA, whole and half states, every CTA and cluster
size, phase tables kept for all layers, refilled per layer and absent, and
circuits deeper than the kernel parameters and the sum groups hold."""
import numpy as np
import pytest

from conftest import (ENERGY_RTOL, GRAD_TOL, angles, assert_state_close, complete_int, gnp_fp,
                      gnp_int)

pytestmark = pytest.mark.gpu

WIDE = 300000  # cut values beyond every phase table


@pytest.mark.parametrize("n,P,kind", [
    (2, 1, "int"), (3, 2, "fp"), (5, 40, "fp"), (7, 33, "int"), (8, 2, "int"), (8, 3, "fp"),
    (9, 1, "int"), (9, 4, "fp"), (10, 2, "wide"), (10, 3, "int"), (11, 1, "fp"), (11, 64, "int"),
    (12, 2, "int"), (12, 3, "fp"), (13, 1, "wide"), (13, 12, "int"), (14, 1, "int"), (14, 2, "fp"),
    (14, 35, "int"), (15, 3, "int"), (15, 2, "wide"), (16, 1, "fp"), (16, 2, "int"),
    (16, 5, "int")])
def test_small_instances(ctx, oracle, n, P, kind):
    rng = np.random.default_rng(3000 * n + P)
    W = {"int": lambda: complete_int(n, rng, -3, 10), "fp": lambda: gnp_fp(n, rng),
         "wide": lambda: gnp_int(n, rng, lo=-WIDE, hi=WIDE)}[kind]()
    g, b = angles(rng, P)
    if kind == "wide":
        g /= WIDE  # keep gamma * W at ordinary size
    b[::3] += np.pi  # both forms of the reduced rotation, and negative factors
    st = ctx.state(n)
    try:
        e = ctx.qaoa_forward(st, W, g, b)
        psi = st.to_host()
    finally:
        st.free()
    want = oracle.qaoa_logical(W, g, b)
    assert_state_close(psi, want, what=f"N={n} P={P} {kind}")
    eo, go, bo = oracle.energy_grad(W, g, b)
    escale = max(1.0, abs(eo), np.abs(W).sum())
    assert abs(e - eo) <= ENERGY_RTOL * escale
    e2, gg, gb = ctx.energy_grad(n, W, g, b)
    scale = max(1.0, np.abs(go).max(), np.abs(bo).max())
    assert abs(e2 - eo) <= ENERGY_RTOL * escale
    assert np.abs(gg - go).max() <= GRAD_TOL * scale
    assert np.abs(gb - bo).max() <= GRAD_TOL * scale
