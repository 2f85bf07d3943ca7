"""The tensor-core DGT against the oracle and the CUDA-core plans: every kernel size, counts
around its units (1, 2 or 4 residues of one prime) and its persistent grid, edge values, the
sources of the inverse, work lists and prescaled tables.  Integer results: equality."""
import numpy as np
import pytest

from tests.common import fold, random_poly_residues, unfold

pytestmark = pytest.mark.gpu

SIZES = (2048, 4096, 8192, 16384, 32768, 65536)


def _engines(gpu, k, nphi, t=256):
    from cupoly_b200.engine import Engine
    e, o = Engine(k, 0, nphi, t), Engine(k, 0, nphi, t)
    e.set_tensor(2)
    o.set_tensor(0)
    assert e.get_tensor() and not o.get_tensor()
    return e, o


@pytest.mark.parametrize("nphi", SIZES)
def test_forward_and_inverse_match_the_oracle(gpu, nphi):
    from cupoly_b200.engine import FORWARD, INVERSE, from_u64, to_u64
    from oracle import coracle
    e, o = _engines(gpu, 2, nphi)
    rows = random_poly_residues(5, e.Q, nphi)
    rows[0, :3] = [0, e.Q[0] - 1, 1]  # the largest and smallest residues
    rows[1, :] = e.Q[1] - 1
    x = from_u64(fold(rows)[None])
    y = x.clone()
    e.dgt(x, 0, FORWARD)
    o.dgt(y, 0, FORWARD)
    assert np.array_equal(to_u64(x), to_u64(y))
    e.dgt(x, 0, INVERSE)
    assert np.array_equal(unfold(to_u64(x))[0], rows)
    # and as a product: the oracle's, coefficient domain
    b = random_poly_residues(6, e.Q, nphi)
    c, ws = e.empty(0), e.polymul_workspace(0, 1)
    e.polymul(c, from_u64(fold(rows)[None]), from_u64(fold(b)[None]), 0, ws)
    assert np.array_equal(unfold(to_u64(c))[0], coracle.polymul(rows[None], b[None], e.Q)[0])
    e.check()


@pytest.mark.parametrize("nphi", SIZES)
@pytest.mark.parametrize("P", (1, 2, 3, 4, 5, 149, 301))
def test_counts_around_units_and_grid(gpu, nphi, P):
    import torch
    from cupoly_b200.engine import FORWARD, INVERSE, QBase
    if P * nphi > 1 << 22:
        pytest.skip("covered by the smaller sizes")
    e, o = _engines(gpu, 3, nphi)
    x = torch.randint(0, 1 << 62, (P, 3, nphi // 2, 2), device="cuda", dtype=torch.int64)
    y = x.clone()
    for direction in (FORWARD, INVERSE, FORWARD):
        e.dgt(x, QBase, direction)
        o.dgt(y, QBase, direction)
        assert torch.equal(x, y)
    e.check()


@pytest.mark.parametrize("nphi, k, P", [(2048, 1, 3), (4096, 2, 5), (8192, 3, 2), (16384, 2, 3), (32768, 2, 2)])
def test_chain_polymul_and_strided_batches(gpu, nphi, k, P):
    import torch
    from cupoly_b200 import _lib
    from cupoly_b200.engine import FORWARD, QBase, _ptr, _stream
    e, o = _engines(gpu, k, nphi)
    ins = [torch.randint(0, 1 << 62, (P, k, nphi // 2, 2), device="cuda", dtype=torch.int64) for _ in range(4)]
    outs = []
    for eng in (e, o):
        c = eng.empty(QBase, 3 * P)
        eng.bfv_mul_batch(c, *ins, P, eng.bfv_mul_batch_workspace(P))
        d = eng.empty(QBase, P)
        eng.polymul(d, ins[0], ins[1], QBase, eng.polymul_workspace(QBase, P))
        # polynomials further apart than their length, and not by a multiple of a residue
        s = torch.zeros(P * (k * (nphi // 2) + 3), 2, device="cuda", dtype=torch.int64)
        for q in range(P):
            s[q * (k * (nphi // 2) + 3):][:k * (nphi // 2)] = ins[0][q].reshape(-1, 2)
        _lib.call("cp_dgt", eng.handle, _ptr(s), QBase, FORWARD, P, k * (nphi // 2) + 3, _stream())
        outs.append((c, d, s))
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    e.check()


@pytest.mark.parametrize("nphi", (2048, 4096, 8192, 16384))
@pytest.mark.parametrize("n", (1, 7, 300, 4097))
def test_work_lists(gpu, nphi, n):
    import torch
    from cupoly_b200 import _lib
    from cupoly_b200.engine import _ptr, _stream
    if n * nphi > 1 << 23:
        n = 601
    e, o = _engines(gpu, 8, nphi)
    g = torch.Generator(device="cuda").manual_seed(n)
    rid = torch.randint(0, 8, (n,), generator=g, device="cuda", dtype=torch.int32)
    a, b = (torch.randint(0, 1 << 62, (n, nphi // 2, 2), generator=g, device="cuda", dtype=torch.int64) for _ in "ab")
    res = []
    for eng in (e, o):
        wa, wb, c, x = (torch.zeros_like(a) for _ in range(4))
        _lib.call("cp_polymul_list", eng.handle, _ptr(c), _ptr(a), _ptr(b), _ptr(wa), _ptr(wb), _ptr(rid), n, _stream())
        x.copy_(a)
        for direction in (0, 1, 0):
            _lib.call("cp_dgt_list", eng.handle, _ptr(x), _ptr(rid), n, direction, _stream())
        res.append((c, x))  # wa and wb are scratch
    for p, q in zip(*res):
        assert torch.equal(p, q)
    e.check()


def test_custom_root_of_i(gpu):
    import torch
    from cupoly_b200.engine import FORWARD, INVERSE, QBase
    e, o = _engines(gpu, 2, 4096)
    xi = [[(p - v) % p for v in pair] for pair, p in zip(e.get_nthroot(), e.primes)]  # (-xi)^N = i, N even
    e.set_nthroot(xi)
    o.set_nthroot(xi)
    assert e.get_tensor()
    x = torch.randint(0, 1 << 62, (3, 2, 2048, 2), device="cuda", dtype=torch.int64)
    y, z = x.clone(), x.clone()
    e.dgt(x, QBase, FORWARD)
    o.dgt(y, QBase, FORWARD)
    assert torch.equal(x, y)
    e.dgt(x, QBase, INVERSE)
    assert torch.equal(x, z)
