"""Coefficient I/O over what its rules let in.  On the tensor cores: cp_crt over B and QB (a column offset into the
matrix, up to six groups of columns), cp_icrt of B and of CKKS bases (a 63-bit prime beside shorter
ones), and wide bases with more tiles than the grid has blocks.  On the CUDA cores: cp_crt on both sides of the
lines between a thread per element and residue and blocks that stage the limbs.  Exact against Python integers."""
import numpy as np
import pytest

from oracle import pyoracle as O
from tests.common import splitmix64, unfold

pytestmark = pytest.mark.gpu


def _limbs(seed, npolys, nphi, nlimbs, modulus):
    w = splitmix64(seed, 5, npolys * nphi * nlimbs).reshape(npolys, nphi, nlimbs)
    w[:, 0] = np.uint64(0xFFFFFFFFFFFFFFFF)
    for at, v in ((1, 0), (2, 1), (3, modulus - 1), (4, modulus), (5, modulus // 2)):
        if v < 1 << (64 * nlimbs):
            w[:, at] = [(v >> (64 * i)) & 0xFFFFFFFFFFFFFFFF for i in range(nlimbs)]
    return w


def _check(e, base, primes, npolys, nphi, nlimbs, polys):
    import torch
    from cupoly_b200.engine import QBBase, from_u64, limbs_to_ints, to_u64
    mod = O.prod(primes)
    w = _limbs(len(primes) * 131 + nlimbs, npolys, nphi, nlimbs, mod)
    x = e.empty(base, npolys)
    e.crt(x, from_u64(w), base)
    ints = {q: limbs_to_ints(w[q]) for q in polys}
    for q in polys:
        res = unfold(to_u64(x[q:q + 1]))[0]
        for r, p in enumerate(primes):
            assert np.array_equal(res[r], np.array([v % p for v in ints[q]], dtype=np.uint64)), (q, r)
    if base != QBBase:
        nl = max(nlimbs, len(primes))
        back = torch.full((npolys, nphi, nl), -1, dtype=torch.int64, device="cuda")
        e.icrt(back, x, base)
        for q in polys:
            assert limbs_to_ints(to_u64(back[q])) == [v % mod for v in ints[q]], q
    e.check()


# tiles x limbs x residues >= 16384 and at most 32 limbs: cp_crt's tensor-core rule
@pytest.mark.parametrize("k,kl,nphi,npolys,nlimbs,base", [
    (5, 6, 2048, 64, 6, 1), (3, 8, 1024, 128, 8, 1), (24, 24, 256, 40, 24, 1), (2, 17, 512, 40, 17, 1),
    (1, 1, 8192, 300, 2, 2), (5, 6, 2048, 64, 5, 2), (4, 13, 512, 60, 17, 2), (24, 24, 256, 20, 32, 2),
    (24, 24, 1024, 40, 24, 2)])
def test_crt_over_every_base(gpu, k, kl, nphi, npolys, nlimbs, base):
    from cupoly_b200.engine import Engine
    e = Engine(k, kl, nphi, 256)
    primes = e.base_primes(base)
    assert npolys * (nphi // 256) * nlimbs * len(primes) >= 16384 and nlimbs <= 32
    _check(e, base, primes, npolys, nphi, nlimbs, sorted({0, npolys // 2, npolys - 1}))


# more tiles than two or four blocks on each SM; from 9 residues on products of 256 columns
@pytest.mark.parametrize("k,nphi,npolys", [(5, 4096, 80), (8, 2048, 90), (9, 2048, 76), (12, 4096, 40), (13, 2048, 77),
                                           (16, 4096, 39)])
def test_bases_with_more_tiles_than_blocks(gpu, k, nphi, npolys):
    from cupoly_b200.engine import Engine
    e = Engine(k, 1, nphi, 256)
    tiles = npolys * (nphi // 256)
    assert tiles > 592 and tiles * k * k >= 16384
    _check(e, 0, e.Q, npolys, nphi, k, [0, npolys // 2, npolys - 1])


@pytest.mark.parametrize("prec", (45, 48, 52, 55))
@pytest.mark.parametrize("k,kl,nphi,npolys,base", [(8, 9, 256, 3, 0), (12, 5, 4096, 40, 0), (16, 2, 512, 2, 0),
                                                   (3, 8, 1024, 150, 1), (5, 2, 4096, 90, 0)])
def test_icrt_of_ckks_bases(gpu, prec, k, kl, nphi, npolys, base):
    from cupoly_b200.engine import Engine
    e = Engine.ckks(k, kl, nphi, prec)
    primes = e.base_primes(base)
    ns, tiles = len(primes), npolys * (nphi // 256)
    assert 5 <= ns <= 16 and (ns >= 8 or tiles * ns * ns >= 32768)  # cp_icrt's tensor-core rule
    _check(e, base, primes, npolys, nphi, ns, sorted({0, npolys // 2, npolys - 1}))


# (prec, k, nphi, polynomials, limbs): blocks of 256 elements x residues around 148, 296, 370 and 407, limb counts
# around 7, 12, 14, 23 and 40 and multiples of 8 and 16, rings below one block, one and two residues, CKKS primes
@pytest.mark.parametrize("prec,k,nphi,npolys,nlimbs", [
    (0, 3, 4, 1, 3), (0, 5, 64, 118, 5), (0, 5, 64, 119, 5), (0, 5, 64, 66, 8), (0, 5, 64, 67, 8), (0, 1, 2048, 40, 7),
    (0, 1, 2048, 40, 8), (0, 1, 8192, 84, 12), (0, 2, 2048, 50, 6), (0, 2, 2048, 52, 6), (0, 4, 1024, 18, 14),
    (0, 4, 1024, 19, 14), (0, 4, 512, 37, 23), (0, 3, 512, 49, 23), (0, 4, 512, 37, 40), (0, 4, 512, 37, 16),
    (0, 4, 2048, 18, 12), (0, 7, 1024, 29, 7), (0, 7, 1024, 30, 7), (0, 2, 8192, 40, 13),
    (55, 2, 64, 3, 40), (55, 4, 512, 3, 4), (55, 4, 512, 3, 8), (55, 8, 512, 19, 16), (45, 6, 2048, 30, 40),
    (48, 6, 1024, 40, 7), (52, 2, 1024, 40, 3)])
def test_crt_on_the_cuda_cores(gpu, prec, k, nphi, npolys, nlimbs):
    from cupoly_b200.engine import Engine
    e = Engine.ckks(k, 1, nphi, prec) if prec else Engine(k, 1, nphi, 256)
    w = _limbs(k * 7 + nlimbs, npolys, nphi, nlimbs, O.prod(e.Q)) if nphi >= 8 else splitmix64(
        3, 5, npolys * nphi * nlimbs).reshape(npolys, nphi, nlimbs)
    from cupoly_b200.engine import from_u64, limbs_to_ints, to_u64
    x = e.empty(0, npolys)
    e.crt(x, from_u64(w), 0)
    got = to_u64(x).reshape(npolys, k, nphi // 2, 2)
    for q in sorted({0, npolys // 2, npolys - 1}):
        ints, res = limbs_to_ints(w[q]), unfold(got[q:q + 1])[0]
        for r, p in enumerate(e.Q):
            assert np.array_equal(res[r], np.array([v % p for v in ints], dtype=np.uint64)), (q, r)


# more primes than are kept in registers (15), where the tensor cores (16 at most, N >= 128) do not take them: rings
# below a block's 64 elements, most limbs, CKKS digits that need a division
@pytest.mark.parametrize("prec,k,kl,nphi,npolys,nlimbs,base", [
    (0, 16, 1, 16, 3, 16, 0), (0, 16, 1, 128, 5, 19, 0), (0, 17, 1, 64, 2, 17, 0), (0, 19, 1, 512, 30, 25, 0),
    (0, 24, 24, 1024, 40, 24, 1), (0, 24, 24, 256, 3, 64, 0), (45, 17, 1, 256, 3, 17, 0), (55, 24, 1, 512, 20, 25, 0),
    (52, 20, 18, 64, 7, 20, 1)])
def test_icrt_of_wide_bases(gpu, prec, k, kl, nphi, npolys, nlimbs, base):
    from cupoly_b200.engine import Engine
    e = Engine.ckks(k, kl, nphi, prec) if prec else Engine(k, kl, nphi, 256)
    _check(e, base, e.base_primes(base), npolys, nphi, nlimbs, sorted({0, npolys // 2, npolys - 1}))
