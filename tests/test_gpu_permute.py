"""GPU qubit permutations in HBM (fq_permute_qubits, fq_swap_blocks) against
numpy, bit for bit: states smaller than a tile and a thread block, whole
tiles and many, permutations that keep, reverse, rotate and shuffle the low
bits (the tile holds the low bits of both sides)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def permuted(v, perm):
    n = len(perm)
    y = np.arange(1 << n)
    x = np.zeros_like(y)
    for b, p in enumerate(perm):
        x |= ((y >> p) & 1) << b
    return v[x]


def on_device(ctx, v, fn, copy=False):
    n = int(np.log2(v.size))
    a = ctx.state(n)
    b = ctx.state(n) if copy else None
    try:
        a.from_host(v)
        fn(a, b)
        return (b if copy else a).to_host()
    finally:
        a.free()
        if copy:
            b.free()


def state(n, rng):
    return rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)


@pytest.mark.parametrize("kind", ["identity", "reverse", "rotate", "shuffle", "swap_low"])
@pytest.mark.parametrize("n", [1, 2, 5, 6, 8, 9, 10, 11, 14, 19])
def test_permute_qubits(ctx, n, kind):
    rng = np.random.default_rng(100 * n)
    ident = np.arange(n)
    perm = {"identity": ident, "reverse": ident[::-1].copy(), "rotate": np.roll(ident, n // 2),
            "shuffle": rng.permutation(n),
            "swap_low": np.concatenate([ident[:2][::-1], ident[2:]])}[kind]
    v = state(n, rng)
    got = on_device(ctx, v, lambda a, b: ctx.permute_qubits(a, b, perm), copy=True)
    assert np.array_equal(got, permuted(v, perm))


@pytest.mark.parametrize("n,out,into,k", [(2, 0, 1, 1), (3, 1, 2, 1), (7, 0, 4, 3), (9, 2, 6, 3),
                                          (12, 0, 6, 6), (13, 7, 10, 3), (16, 0, 14, 2),
                                          (18, 3, 11, 7)])
def test_swap_blocks(ctx, n, out, into, k):
    perm = np.arange(n)
    perm[out:out + k], perm[into:into + k] = np.arange(into, into + k), np.arange(out, out + k)
    v = state(n, np.random.default_rng(n))
    got = on_device(ctx, v, lambda a, b: ctx.swap_blocks(a, out, into, k))
    assert np.array_equal(got, permuted(v, perm))
