"""Gaussian products and dot products with the two-sum accumulators: edge residues, the largest
number of terms, primes of both forms, against Python integers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gauss_mul(a, b, p):
    return (a[0] * b[0] - a[1] * b[1]) % p, (a[0] * b[1] + a[1] * b[0]) % p


@pytest.mark.parametrize("ckks", (0, 55))
@pytest.mark.parametrize("terms", (1, 2, 5, 64))
def test_products_and_dots_at_edges(gpu, ckks, terms):
    from cupoly_b200.engine import Engine, QBase, from_u64, to_u64
    e = Engine(3, 0, 64, 256, ckks_prec=ckks)
    N, n = e.N, terms
    rng = np.random.default_rng(terms + ckks)

    def poly(i):
        x = np.zeros((3, N, 2), dtype=np.uint64)
        for r, p in enumerate(e.Q):
            edge = [0, 1, p - 1, p // 2, p // 2 + 1, (1 << 32) % p, ((1 << 32) - 1) % p, (1 << 62) % p]
            x[r] = rng.integers(0, p, size=(N, 2), dtype=np.uint64)
            x[r, :8] = [[edge[j], edge[(3 * j + i) % 8]] for j in range(8)]
            x[r, 8] = p - 1  # every product and sum at its largest
            x[r, 9] = [p - 1, 0] if i % 2 else [0, p - 1]
        return x

    a, b = [poly(i) for i in range(n)], [poly(i + 1) for i in range(n)]
    da, db = [from_u64(x[None]) for x in a], [from_u64(x[None]) for x in b]
    want = np.zeros((3, N, 2), dtype=np.uint64)
    for r, p in enumerate(e.Q):
        for j in range(N):
            s = [0, 0]
            for t in range(n):
                z = _gauss_mul([int(v) for v in a[t][r, j]], [int(v) for v in b[t][r, j]], p)
                s = [(s[0] + z[0]) % p, (s[1] + z[1]) % p]
            want[r, j] = s
    c = e.empty(QBase)
    e.dot(c, da, db, QBase)
    assert np.array_equal(to_u64(c)[0], want)
    import torch
    e.dot_batch(c, torch.cat(da), torch.cat(db), n, 1, QBase)
    assert np.array_equal(to_u64(c)[0], want)
    if n == 1:
        e.mul(c, da[0], db[0], QBase)
        assert np.array_equal(to_u64(c)[0], want)
        e.muladd(c, da[0], db[0], da[0], QBase)
        P = np.array(e.Q, dtype=np.uint64)[:, None, None]
        assert np.array_equal(to_u64(c)[0], (want + a[0]) % P)
    if n == 2:
        o = [e.empty(QBase) for _ in range(3)]
        e.dr2(*o, da[0], da[1], db[1], db[0], QBase)  # c1 = a0 b0 + a1 b1
        assert np.array_equal(to_u64(o[1])[0], want)
