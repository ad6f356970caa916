"""Phases of integer weights on the engine's passes against 80-bit arithmetic
(numpy's long double): 20 qubits, complete graphs, cut values up to a
thousand.

Tolerances.  A layer takes 20 rotations and a phase of eight factors, each
rounded to about 2^-53, and the power of the rotations' common factor: some
60 roundings, 2 * 60 * 2^-53 = 1.4e-14 for two layers at the very most, if
all add up.  An angle gamma * C that is rounded before its sine is off by up
to pi * 1000 * 2^-53 = 3.5e-13 on top, for all amplitudes of that cut value.
An entry of the gradient turns an angle's error d into at most d * sum|w|
relative to <C>'s scale, and into less for random signs: as for the state, with
<C> in the place of the norm."""
import numpy as np
import pytest

from conftest import angles, complete_int

pytestmark = pytest.mark.gpu

TOL = 1.4e-14
LD = np.longdouble


def rotate(v, q, beta):
    re, im = (x.reshape(-1, 2, 1 << q) for x in v)
    c, s = np.cos(LD(beta) / 2), np.sin(LD(beta) / 2)
    ar, ai, br, bi = re[:, 0], im[:, 0], re[:, 1], im[:, 1]
    ar, ai, br, bi = c * ar + s * bi, c * ai - s * br, c * br + s * ai, c * bi - s * ar
    re[:, 0], im[:, 0], re[:, 1], im[:, 1] = ar, ai, br, bi


def phase(v, cut, total, gamma):
    c = np.arange(int(total) + 1)
    x = (2 * c - total).astype(LD) * LD(gamma) / 2
    cs, sn = np.cos(x)[cut], np.sin(x)[cut]
    v[0], v[1] = v[0] * cs - v[1] * sn, v[0] * sn + v[1] * cs


def truth(W, gammas, betas):
    """State, <C>, dE/dgamma, dE/dbeta in long double."""
    n, total = W.shape[0], W.sum()
    z = np.arange(1 << n)
    cut = np.zeros(1 << n, dtype=np.int64)
    for i in range(n):
        for j in range(i + 1, n):
            cut += int(W[i, j]) * (((z >> i) ^ (z >> j)) & 1)
    psi = [np.full(1 << n, np.sqrt(LD(2)) ** -n), np.zeros(1 << n, dtype=LD)]
    for g, b in zip(gammas, betas):
        phase(psi, cut, total, g)
        for q in range(n):
            rotate(psi, q, b)
    state = [x.copy() for x in psi]
    e = ((psi[0] ** 2 + psi[1] ** 2) * cut).sum()
    lam = [x * cut for x in psi]
    gg, gb = np.zeros(len(gammas), dtype=LD), np.zeros(len(gammas), dtype=LD)
    for k in reversed(range(len(gammas))):
        for q in range(n):
            re, im = (x.reshape(-1, 2, 1 << q)[:, ::-1].reshape(-1) for x in psi)
            gb[k] += (lam[0] * im - lam[1] * re).sum()
        for v in (psi, lam):
            for q in range(n):
                rotate(v, q, -betas[k])
        gg[k] = -((lam[0] * psi[1] - lam[1] * psi[0]) * (2 * cut - int(total))).sum()
        for v in (psi, lam):
            phase(v, cut, total, -gammas[k])
    return state, e, gg, gb


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_integer_phases_are_as_exact_as_the_rotations(ctx, seed):
    n, P = 20, 2
    rng = np.random.default_rng([seed, n])
    W, (g, b) = complete_int(n, rng), angles(rng, P)
    (re, im), e, gg, gb = truth(W, g, b)
    st = ctx.state(n)
    try:
        got = ctx.qaoa_forward(st, W, g, b)
        psi = st.to_host()
    finally:
        st.free()
    diff = np.sqrt(((psi.real - re) ** 2 + (psi.imag - im) ** 2).sum())
    assert float(diff) <= TOL
    e2, dg, db = ctx.energy_grad(n, W, g, b)
    assert abs(float(got - e)) <= TOL * float(e) and abs(float(e2 - e)) <= TOL * float(e)
    assert float(np.abs(db - gb).max()) <= TOL * float(e)
    assert float(np.abs(dg - gg).max()) <= TOL * float(e)


@pytest.mark.parametrize("gamma", [3e7, -4e9, 3.7e12, 1e18, 1e30])
def test_large_angles(ctx, gamma):
    """Far beyond 2^26 the rounding of gamma * C is no small angle: the
    phases are those of the exact product (11 and 53 bits: long double holds
    it) and the norm is kept."""
    n = 20
    rng = np.random.default_rng(n)
    W, b = complete_int(n, rng), 0.7
    z = np.arange(1 << n)
    cut = np.zeros(1 << n, dtype=np.int64)
    for i in range(n):
        for j in range(i + 1, n):
            cut += int(W[i, j]) * (((z >> i) ^ (z >> j)) & 1)
    v = [np.full(1 << n, np.sqrt(LD(2)) ** -n), np.zeros(1 << n, dtype=LD)]
    phase(v, cut, W.sum(), gamma)
    for q in range(n):
        rotate(v, q, b)
    st = ctx.state(n)
    try:
        ctx.qaoa_forward(st, W, [gamma], [b])
        psi = st.to_host()
    finally:
        st.free()
    assert float(np.sqrt(((psi.real - v[0]) ** 2 + (psi.imag - v[1]) ** 2).sum())) <= TOL / 2
